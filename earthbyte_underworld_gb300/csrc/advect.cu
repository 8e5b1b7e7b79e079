// Material-point advection on the device: the SwarmAdvector time integration of the particle
// coordinates with the current velocity solution.
//
// Reference (paths relative to the Underworld 1.x tree):
//   time derivative   PICellerator/MaterialPoints/src/SwarmAdvector.c:288-314: the velocity
//                     interpolated at the point (FieldVariable_InterpolateValueAt ->
//                     StgFEM/Discretisation/src/FeVariable.c:773-800); a point outside the mesh
//                     has no velocity
//   first order       StgDomain/Utils/src/TimeIntegrand.c:221-265: x = x0 + dt v(x0)
//   second order      TimeIntegrand.c:267-337: predictor x0 + dt/2 v(x0), corrector
//                     x0 + dt v(predictor); a predictor outside the mesh falls back to the
//                     first-order update when allowFallbackToFirstOrder is set, else stops
//   ownership         SwarmAdvector_AdvectionFinish -> Swarm_UpdateAllParticleOwners
//                     (SwarmAdvector.c:375-382): here the next uwgpu_bin_and_map
//
// Points are independent (the reference keeps each point's start value before its predictor),
// so the update is one thread per point: element search with the mapper's tie rules (locate.cuh), the
// closed form local coordinate of the affine element, Q1 shape functions on the SoA nodal velocity.
// All points are written to a second coordinate set, which replaces the first only when every
// point succeeded, so a failed step leaves the swarm as it was.
#include <cmath>
#include <cstring>
#include <string>
#include <utility>

#include "internal.cuh"
#include "locate.cuh"

namespace uwg {

namespace {

struct AdvMesh {
    AxisMap ax[3];
    const double* h[3];   // per axis: x0[nel], then h[nel], then 1/h[nel] (binning.cu)
    int64_t nnx, nny, nn;
};

// velocity at point x: Q1 interpolation of the SoA nodal velocity u[d][node].  The fixed-point element
// search and the stored reciprocal widths leave about 50 FP64 instructions (24 FMAs of them the sum over the
// corners); with divisions for the element, the node coordinates and the local coordinate it was over 200,
// and the kernel is bound by FP64 (1.73M points, second order: 1,590 us before).
template <int DIM>
__device__ __forceinline__ bool velocity_at(const AdvMesh& m, const double* __restrict__ u, const double x[3],
                                            double v[3]) {
    int ie[3] = {0, 0, 0};
    double f[3][2];   // linear shape functions of the two nodes per axis
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        if (!axis_index(m.ax[d], x[d], ie[d])) return false;
        const int nel = m.ax[d].nel;
        f[d][1] = (x[d] - __ldg(m.h[d] + ie[d])) * __ldg(m.h[d] + 2 * nel + ie[d]);
        f[d][0] = 1.0 - f[d][1];
    }
    const int64_t base = ie[0] + m.nnx * (ie[1] + m.nny * (int64_t)ie[2]);
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = 0.0;
#pragma unroll
    for (int b = 0; b < (1 << (DIM - 1)); ++b) {   // corners by pairs along x
        double g = f[1][b & 1];
        if (DIM == 3) g *= f[2][b >> 1];
        const int64_t node = base + (b & 1) * m.nnx + (DIM == 3 ? (b >> 1) * m.nnx * m.nny : 0);
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const double N = g * f[0][a];
#pragma unroll
            for (int d = 0; d < DIM; ++d) v[d] = fma(N, __ldg(u + (int64_t)d * m.nn + node + a), v[d]);
        }
    }
    return true;
}

// counters: [0] points without a velocity (start or, without fallback, predictor outside the
// mesh), [1] first-order fallbacks, [2] points that end outside the mesh
template <int DIM>
__global__ void k_advect(int64_t np, const __grid_constant__ AdvMesh m, const double* __restrict__ u, double dt, int order, int fallback,
                         const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
                         double* __restrict__ qx, double* __restrict__ qy, double* __restrict__ qz,
                         uint32_t* __restrict__ counters) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const double x0[3] = {px[p], py[p], DIM == 3 ? pz[p] : 0.0};
    double v0[3] = {0, 0, 0}, v1[3] = {0, 0, 0}, x1[3] = {x0[0], x0[1], x0[2]};
    bool ok = velocity_at<DIM>(m, u, x0, v0);
    if (ok) {
        if (order == 1) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) x1[d] = x0[d] + dt * v0[d];
        } else {
            double xm[3] = {x0[0], x0[1], x0[2]};
#pragma unroll
            for (int d = 0; d < DIM; ++d) xm[d] = x0[d] + 0.5 * dt * v0[d];
            if (velocity_at<DIM>(m, u, xm, v1)) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) x1[d] = x0[d] + dt * v1[d];
            } else if (fallback) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) x1[d] = x0[d] + dt * v0[d];
                atomicAdd(&counters[1], 1u);
            } else {
                ok = false;
            }
        }
    }
    if (!ok) {
        atomicAdd(&counters[0], 1u);
    } else {
        int dummy;
        bool inside = true;
#pragma unroll
        for (int d = 0; d < DIM; ++d) inside = inside && axis_index(m.ax[d], x1[d], dummy);
        if (!inside) atomicAdd(&counters[2], 1u);
    }
    qx[p] = x1[0];
    qy[p] = x1[1];
    if (DIM == 3) qz[p] = x1[2];
}

}  // namespace

void advect_particles(Context& c, double dt, int order, bool fallback, uint32_t& fell_back, uint32_t& left_mesh) {
    UWG_REQUIRE(c.has_points, UWGPU_ERR_STATE, "advection requested before particles_upload");
    UWG_REQUIRE(c.has_solution, UWGPU_ERR_STATE, "advection requested before a velocity solution");
    UWG_REQUIRE(order == 1 || order == 2, UWGPU_ERR_ARGUMENT, "advection order must be 1 or 2");
    UWG_REQUIRE(std::isfinite(dt), UWGPU_ERR_ARGUMENT, "dt must be finite");
    const MeshDesc& md = c.mesh;
    AdvMesh m;
    for (int d = 0; d < 3; ++d) m.ax[d] = axis_map(md.min[d], md.max[d], md.nel[d]);
    axis_tables(c, m.h);
    m.nnx = md.nnx;
    m.nny = md.nny;
    m.nn = md.nn;
    const int64_t np = c.np;
    c.qx.ensure((size_t)(np > 0 ? np : 1));
    c.qy.ensure((size_t)(np > 0 ? np : 1));
    if (md.dim == 3) c.qz.ensure((size_t)(np > 0 ? np : 1));
    c.err_count.ensure(4);
    UWG_CUDA(cudaMemsetAsync(c.err_count.p, 0, 4 * sizeof(uint32_t), c.stream));
    if (np > 0) {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        if (md.dim == 3)
            k_advect<3><<<blocks_for(np, 256), 256, 0, c.stream>>>(np, m, c.u_sol.p, dt, order, fallback ? 1 : 0, c.px.p,
                                                                   c.py.p, c.pz.p, c.qx.p, c.qy.p, c.qz.p, c.err_count.p);
        else
            k_advect<2><<<blocks_for(np, 256), 256, 0, c.stream>>>(np, m, c.u_sol.p, dt, order, fallback ? 1 : 0, c.px.p,
                                                                   c.py.p, nullptr, c.qx.p, c.qy.p, nullptr, c.err_count.p);
        note_work(c, UWGPU_KERNEL_BINNING, (double)np * md.dim * 16.0, (double)np * 80.0);
    }
    check_launch("k_advect");
    uint32_t counters[4] = {0, 0, 0, 0};
    UWG_CUDA(cudaMemcpyAsync(c.host_scalars, c.err_count.p, sizeof(counters), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    std::memcpy(counters, c.host_scalars, sizeof(counters));
    if (counters[0] > 0)
        throw Error(UWGPU_ERR_DOMAIN, std::to_string(counters[0]) +
                                          " material points have no velocity (outside the mesh); the swarm is unchanged");
    c.px.swap(c.qx);
    c.py.swap(c.qy);
    if (md.dim == 3) {
        c.pz.swap(c.qz);
    }
    c.mapped = false;   // ownership changes: the next bin_and_map rebuilds the cell tables
    fell_back = counters[1];
    left_mesh = counters[2];
}

}  // namespace uwg
