// Material point -> element binning and the integration-point mapper.
//
// Reference behaviour (paths relative to the Underworld 1.x tree):
//   element search   StgDomain/Mesh/src/Mesh_RegularAlgorithms.c:194-226 (sep from :154-175,
//                    Num_Approx epsilon 1e-12 from StGermain/Base/Foundation/src/Numerics.c:37-41)
//   cell tables      PICellerator/MaterialPoints/src/CoincidentMapper.c:176-242 appends points in
//                    ascending index order (StgDomain/Swarm/src/SwarmClass.c:1155-1184)
//   local coords     StgFEM/Discretisation/src/ElementType.c:227-350 (Newton; on the affine
//                    elements of a regular mesh it reproduces the closed form used here)
//
// GPU design: counting sort with integer atomics on HBM-resident counts (the count an atomic returns is
// the point's place in its element, so the scatter needs no second atomic), an exclusive scan,
// an unordered scatter, then one warp per element ranks its points by index so the final
// permutation equals the reference's append order exactly.  The same warp computes xi and
// gathers the per-point inputs into slot order (SoA), so assembly reads them coalesced.
#include <cstring>

#include "internal.cuh"
#include "locate.cuh"

namespace uwg {

struct MeshParams {
    AxisMap ax[3];
    const double* tab[3];   // per axis: lower node x0[nel], width h[nel], 1/h[nel] of every element layer
};

// x0, h, RN(1/h) of the element layers of one axis
__global__ void k_axis_table(int nel, double mn, double mx, double* __restrict__ tab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nel) return;
    const double x0 = node_coord_1d(i, nel, mn, mx), x1 = node_coord_1d(i + 1, nel, mn, mx);
    const double h = x1 - x0;
    tab[i] = x0;
    tab[nel + i] = h;
    tab[2 * nel + i] = __drcp_rn(h);
}

void axis_tables(Context& c, const double* tab[3]) {
    const MeshDesc& m = c.mesh;
    int64_t off[3], total = 0;
    for (int d = 0; d < 3; ++d) {
        off[d] = d < m.dim ? total : 0;
        if (d < m.dim) total += 3 * (int64_t)m.nel[d];
    }
    if (!c.axis_tab_ok) {   // once per mesh
        c.axis_tab.ensure((size_t)total);
        for (int d = 0; d < m.dim; ++d) {
            LaunchScope ls(c, UWGPU_KERNEL_BINNING);
            k_axis_table<<<blocks_for(m.nel[d], 128), 128, 0, c.stream>>>(m.nel[d], m.min[d], m.max[d], c.axis_tab.p + off[d]);
        }
        check_launch("k_axis_table");
        c.axis_tab_ok = true;
    }
    for (int d = 0; d < 3; ++d) tab[d] = c.axis_tab.p + off[d];
}

static MeshParams params_of(Context& c) {
    MeshParams p;
    for (int d = 0; d < 3; ++d) p.ax[d] = axis_map(c.mesh.min[d], c.mesh.max[d], c.mesh.nel[d]);
    axis_tables(c, p.tab);
    return p;
}

// element of every point, its place in the element (in the order of the atomics) and the counts
template <int DIM>
__global__ void k_locate(int64_t np, const double* __restrict__ px, const double* __restrict__ py,
                         const double* __restrict__ pz, const __grid_constant__ MeshParams mp, uint32_t* __restrict__ cell,
                         uint32_t* __restrict__ place, uint32_t* __restrict__ counts, uint32_t* __restrict__ err) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const double pt[3] = {px[p], py[p], DIM == 3 ? pz[p] : 0.0};
    unsigned e = 0, mul = 1;
    bool ok = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        int i = 0;
        ok = axis_index(mp.ax[d], pt[d], i) && ok;
        e += mul * (unsigned)i;
        mul *= (unsigned)mp.ax[d].nel;
    }
    if (!ok) {
        cell[p] = 0xffffffffu;
        atomicAdd(err, 1u);
        return;
    }
    cell[p] = e;
    place[p] = atomicAdd(&counts[e], 1u);
}

// ---- exclusive scan of u32 counts: out[0..n] with out[n] = total ----
constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem_warp, uint32_t& total) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? smem_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) smem_warp[lane] = w;
    }
    __syncthreads();
    uint32_t warp_prefix = warp ? smem_warp[warp - 1] : 0u;
    total = smem_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

__global__ void k_scan_tiles(int64_t n, const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                             uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t sw[32];
    int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = (base + i < n) ? in[base + i] : 0u;
        s += v[i];
    }
    uint32_t total;
    uint32_t pre = block_exclusive_scan(s, sw, total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (base + i < n) out[base + i] = pre;
        pre += v[i];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Single block: exclusive scan of the tile sums in chunks, carrying the running total.
__global__ void k_scan_tile_sums(int64_t ntiles, uint32_t* __restrict__ tile_sums, uint32_t* __restrict__ grand) {
    __shared__ uint32_t sw[32];
    uint32_t carry = 0;
    for (int64_t base = 0; base < ntiles; base += blockDim.x) {
        int64_t i = base + threadIdx.x;
        uint32_t v = i < ntiles ? tile_sums[i] : 0u;
        uint32_t total;
        uint32_t pre = block_exclusive_scan(v, sw, total);
        if (i < ntiles) tile_sums[i] = carry + pre;
        carry += total;
    }
    if (threadIdx.x == 0) *grand = carry;
}

__global__ void k_scan_add(int64_t n, uint32_t* __restrict__ out, const uint32_t* __restrict__ tile_sums) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += tile_sums[i / kScanTile];
}

// The whole scan in one block, for the element counts of small meshes (one launch of 2 us instead of three)
constexpr int64_t kScanSmall = 2 * 1024 * kScanItems;

__global__ void __launch_bounds__(1024) k_scan_small(int64_t n, const uint32_t* __restrict__ in, uint32_t* __restrict__ out) {
    __shared__ uint32_t sw[32];
    uint32_t carry = 0;
    for (int64_t t = 0; t < n; t += 1024 * kScanItems) {
        const int64_t base = t + (int64_t)threadIdx.x * kScanItems;
        uint32_t v[kScanItems], s = 0, total;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            v[i] = (base + i < n) ? in[base + i] : 0u;
            s += v[i];
        }
        uint32_t pre = carry + block_exclusive_scan(s, sw, total);
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            if (base + i < n) out[base + i] = pre;
            pre += v[i];
        }
        carry += total;
    }
    if (threadIdx.x == 0) out[n] = carry;
}

static void exclusive_scan(Context& c, const uint32_t* in, uint32_t* out, int64_t n) {
    if (n <= kScanSmall) {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        k_scan_small<<<1, 1024, 0, c.stream>>>(n, in, out);
        check_launch("k_scan_small");
        return;
    }
    int64_t ntiles = (n + kScanTile - 1) / kScanTile;
    if (ntiles < 1) ntiles = 1;
    c.block_sums.ensure((size_t)ntiles);
    {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        k_scan_tiles<<<(unsigned)ntiles, kScanThreads, 0, c.stream>>>(n, in, out, c.block_sums.p);
    }
    check_launch("k_scan_tiles");
    {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        k_scan_tile_sums<<<1, 1024, 0, c.stream>>>(ntiles, c.block_sums.p, out + n);
    }
    check_launch("k_scan_tile_sums");
    {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        k_scan_add<<<blocks_for(n, 256), 256, 0, c.stream>>>(n, out, c.block_sums.p);
    }
    check_launch("k_scan_add");
}

__global__ void k_scatter(int64_t np, const uint32_t* __restrict__ cell, const uint32_t* __restrict__ place,
                          const uint32_t* __restrict__ offsets, uint32_t* __restrict__ tmp_perm) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const uint32_t e = cell[p];
    if (e == 0xffffffffu) return;
    tmp_perm[offsets[e] + place[p]] = (uint32_t)p;
}

// One warp per element: rank the element's points by point index (the append order of the
// reference cell table), write the permutation, then map every point of the element.
// xi = RN((2 (x - x0) - h) / h): the division by h is a product with RN(1/h) and one FMA correction, which
// gives the correctly rounded quotient (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990): 5 FP64 instructions per axis where two divisions for
// the node coordinates and one for xi took over 30, which bound this kernel (2.4M points: 556 us before).
template <int DIM>
__global__ void __launch_bounds__(256) k_sort_map(int64_t ne, int64_t nslots, const __grid_constant__ MeshParams mp,
                                                  const uint32_t* __restrict__ offsets,
                                                  const uint32_t* __restrict__ tmp_perm, uint32_t* __restrict__ perm,
                                                  const double* __restrict__ px, const double* __restrict__ py,
                                                  const double* __restrict__ pz, const int32_t* __restrict__ pmat,
                                                  const double* __restrict__ peta, const double* __restrict__ prho,
                                                  double* __restrict__ sxi, int32_t* __restrict__ smat,
                                                  double* __restrict__ seta, double* __restrict__ srho) {
    const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (e >= ne) return;
    const uint32_t beg = offsets[e], n = offsets[e + 1] - beg;
    double x0[3], h[3], rh[3];
    unsigned q = (unsigned)e;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const int nel = mp.ax[d].nel;
        const int i = d + 1 < DIM ? (int)(q % (unsigned)nel) : (int)q;
        q /= (unsigned)nel;
        x0[d] = __ldg(mp.tab[d] + i);
        h[d] = __ldg(mp.tab[d] + nel + i);
        rh[d] = __ldg(mp.tab[d] + 2 * nel + i);
    }
    for (uint32_t i0 = 0; i0 < n; i0 += 32) {
        const bool mine = i0 + lane < n;
        const uint32_t v = mine ? tmp_perm[beg + i0 + lane] : 0xffffffffu;
        uint32_t rank = 0;
        for (uint32_t j0 = 0; j0 < n; j0 += 32) {
            const uint32_t w = j0 == i0 ? v : (j0 + lane < n ? tmp_perm[beg + j0 + lane] : 0xffffffffu);
#pragma unroll
            for (int j = 0; j < 32; ++j) rank += __shfl_sync(0xffffffffu, w, j) < v ? 1u : 0u;
        }
        if (!mine) continue;
        const uint32_t slot = beg + rank;
        const double x[3] = {px[v], py[v], DIM == 3 ? pz[v] : 0.0};
        perm[slot] = v;
        smat[slot] = pmat[v];
        if (seta) seta[slot] = peta[v];
        if (srho) srho[slot] = prho[v];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double a = fma(2.0, x[d] - x0[d], -h[d]);
            const double t = a * rh[d];
            sxi[(int64_t)d * nslots + slot] = fma(fma(-t, h[d], a), rh[d], t);
        }
    }
}

void bin_and_map(Context& c) {
    UWG_REQUIRE(c.has_mesh, UWGPU_ERR_STATE, "mesh not set");
    UWG_REQUIRE(c.has_points, UWGPU_ERR_STATE, "material points not uploaded");
    const int64_t np = c.np, ne = c.mesh.ne;
    const MeshParams mp = params_of(c);
    c.cell.ensure((size_t)np);
    c.counts.ensure((size_t)ne + 1);   // and the number of points outside
    c.place.ensure((size_t)np);
    c.offsets.ensure((size_t)ne + 1);
    c.perm.ensure((size_t)np);
    c.tmp_perm.ensure((size_t)np);
    c.sxi.ensure((size_t)np * c.mesh.dim);
    c.smat.ensure((size_t)np);
    c.seta_out.ensure((size_t)np);
    if (c.has_peta) c.seta_in.ensure((size_t)np);
    if (c.has_prho) c.srho_in.ensure((size_t)np);
    uint32_t* err = c.counts.p + ne;
    UWG_CUDA(cudaMemsetAsync(c.counts.p, 0, (ne + 1) * sizeof(uint32_t), c.stream));
    {
        // algorithmic bytes of the whole binning pass: per point coordinates read twice (locate,
        // map), cell id and place written/read, count atomics, unordered and final permutation,
        // material in, xi and material out (+ optional per-point inputs); per element counts
        // and offsets
        int dim = c.mesh.dim;
        double extra = (c.has_peta ? 16.0 : 0.0) + (c.has_prho ? 16.0 : 0.0);
        double per_point = 2 * dim * 8.0 + 16.0 + 16.0 + 12.0 + 8.0 + dim * 8.0 + extra;
        note_work(c, UWGPU_KERNEL_BINNING, per_point * np + 16.0 * ne, 0.0);
    }
    if (np > 0) {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        if (c.mesh.dim == 3)
            k_locate<3><<<blocks_for(np, 256), 256, 0, c.stream>>>(np, c.px.p, c.py.p, c.pz.p, mp, c.cell.p, c.place.p, c.counts.p, err);
        else
            k_locate<2><<<blocks_for(np, 256), 256, 0, c.stream>>>(np, c.px.p, c.py.p, nullptr, mp, c.cell.p, c.place.p, c.counts.p, err);
    }
    check_launch("k_locate");
    exclusive_scan(c, c.counts.p, c.offsets.p, ne);
    if (np > 0) {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        k_scatter<<<blocks_for(np, 256), 256, 0, c.stream>>>(np, c.cell.p, c.place.p, c.offsets.p, c.tmp_perm.p);
    }
    check_launch("k_scatter");
    {
        LaunchScope ls(c, UWGPU_KERNEL_BINNING);
        unsigned blocks = blocks_for(ne * 32, 256);
        double* seta = c.has_peta ? c.seta_in.p : nullptr;
        double* srho = c.has_prho ? c.srho_in.p : nullptr;
        if (c.mesh.dim == 3)
            k_sort_map<3><<<blocks, 256, 0, c.stream>>>(ne, np, mp, c.offsets.p, c.tmp_perm.p, c.perm.p, c.px.p, c.py.p,
                                                       c.pz.p, c.pmat.p, c.peta.p, c.prho.p, c.sxi.p, c.smat.p, seta, srho);
        else
            k_sort_map<2><<<blocks, 256, 0, c.stream>>>(ne, np, mp, c.offsets.p, c.tmp_perm.p, c.perm.p, c.px.p, c.py.p,
                                                       nullptr, c.pmat.p, c.peta.p, c.prho.p, c.sxi.p, c.smat.p, seta, srho);
    }
    check_launch("k_sort_map");
    UWG_CUDA(cudaMemcpyAsync(c.host_scalars, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    uint32_t outside = 0;
    std::memcpy(&outside, c.host_scalars, sizeof(outside));
    c.mapped = true;
    c.assembled = false;
    if (outside)
        throw Error(UWGPU_ERR_DOMAIN, std::to_string(outside) + " material points lie outside the mesh");
}

}  // namespace uwg
