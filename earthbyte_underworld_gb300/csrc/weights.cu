// Discrete Voronoi cell weights of the integration points (PICellerator/Weights/src/DVCWeights.c),
// one warp per element.
//
// The element's local square / cube [-1, 1]^dim carries a fixed grid of res[0] x res[1] (x res[2])
// cells, x fastest, at most 1024 cells: cell c is bit (c & 31) of word (c >> 5), and lane l of
// the warp holds word l of every cell set.  Every point first claims the cell that holds it (a
// later point in the same cell takes it over).  Then the points grow their regions in passes, in
// point order, as the reference does (_DVCWeights_CreateVoronoi, DVCWeights.c:668-714):
//   claim   (_DVCWeights_ClaimCells, :261-317): every cell of the point's boundary set is taken
//           when free, or when held by another point that is farther from the cell's centre
//           (_DVCWeights_DistanceTest, :604-609, evaluated in the same operation order with
//           round-to-nearest intrinsics, so the contest is decided exactly as in FP64 C);
//   update  (_DVCWeights_UpdateBchain, :395-446): the new boundary set is the face neighbours of
//           the cells just taken that the point does not hold (bit shifts of the 1024-bit set
//           across the lanes, with row and plane masks so that no shift wraps around the grid).
// The cells a point tries in one claim are distinct and each decision reads only that cell's
// owner, so processing a boundary set in parallel gives the reference's sequential result.
// Passes end when one takes no cell (each cell changes owner only to a strictly nearer point, so
// the count of passes is bounded; a cap of cells x points + 2 passes flags an error).  Weight =
// cells held x cell volume; new local coordinate = mean of the held cells' centres, summed in
// cell order (_DVCWeights_GetCentroids, :203-231), lane j accumulating point j.
// An element's owners (one byte a cell) and boundary sets live in the warp's shared memory, up to kDvcCap
// points (k_dvc); elements with more points take k_dvc_large, which keeps the sets in a per-slot scratch
// array and is otherwise the plain form.  What bounded the plain form is FP64 (64 cycles a warp instruction
// and scheduler): 17 instructions per contest, and the centroid sums, where each cell's three additions had
// one lane active.  k_dvc decides a contest in FP32 and repeats it in FP64 only when the FP32 value is within
// its error bound of zero, and in the centroid sums every lane walks its own point's cells, so all lanes add
// at once.  13,824 elements of 20 points on 10^3 cells: 11.4 ms before.
#include <algorithm>
#include <cstring>

#include "internal.cuh"

namespace uwg {

namespace {

constexpr int kDvcWarps = 4;
constexpr int kDvcFast = 8;      // warps per block of k_dvc: 88 KB of shared memory, two blocks per SM
constexpr int kDvcCap = 64;      // points per element it takes
constexpr int kDvcPitch = 33;    // words between the points' sets: lanes reading one word of 32 sets do not collide

struct DvcArgs {
    int dim, nx, ny, nz, nc;
    double cen[3][32];   // cell centres per axis (accumulated as in _DVCWeights_ConstructGrid)
    double h[3];         // cell widths 2 / res
    double da;           // cell volume
    int64_t ne, nslots;
    const uint32_t* offsets;
    const double* sxi;   // [d][slot]
    double* oxi;         // [d][slot]
    double* ow;          // [slot]
    uint32_t* bnd;       // [slot][32]
    uint32_t* err;       // [0] elements whose passes hit the cap, [1] elements of more than kDvcCap points
};

__device__ __forceinline__ uint32_t shl_set(uint32_t w, int s, int lane) {
    // bit c of the result = bit c - s of the set
    const int q = s >> 5, r = s & 31;
    uint32_t a = __shfl_up_sync(0xffffffffu, w, q);
    uint32_t b = __shfl_up_sync(0xffffffffu, w, q + 1);
    a = lane >= q ? a : 0u;
    b = lane >= q + 1 ? b : 0u;
    return r ? (a << r) | (b >> (32 - r)) : a;
}

__device__ __forceinline__ uint32_t shr_set(uint32_t w, int s, int lane) {
    // bit c of the result = bit c + s of the set
    const int q = s >> 5, r = s & 31;
    uint32_t a = __shfl_down_sync(0xffffffffu, w, q);
    uint32_t b = __shfl_down_sync(0xffffffffu, w, q + 1);
    a = lane + q < 32 ? a : 0u;
    b = lane + q + 1 < 32 ? b : 0u;
    return r ? (a >> r) | (b << (32 - r)) : a;
}

// (x1 + x2 - x0 - x0)(x1 - x2) + (y1 + y2 - y0 - y0)(y1 - y2) [+ z term], left to right
__device__ __forceinline__ double dvc_contest(int dim, const double c0[3], const double p1[3], const double p2[3]) {
    double t = 0.0;
    for (int d = 0; d < dim; ++d) {
        const double a = __dsub_rn(__dsub_rn(__dadd_rn(p1[d], p2[d]), c0[d]), c0[d]);
        const double v = __dmul_rn(a, __dsub_rn(p1[d], p2[d]));
        t = d == 0 ? v : __dadd_rn(t, v);
    }
    return t;
}

struct DvcWarp {
    uint32_t own[256];                    // owner bytes: cell 32 l + k in byte k & 3 of word 32 (k >> 2) + l; 255: free
    uint32_t set[kDvcCap * kDvcPitch];    // boundary sets, then the points' cells
    float px[3][kDvcCap];
};

__global__ void __launch_bounds__(32 * kDvcFast, 2) k_dvc(const __grid_constant__ DvcArgs a) {
    extern __shared__ __align__(16) unsigned char dvc_smem[];
    __shared__ uint32_t s_cell[1024];     // x, y, z of a cell, a byte each
    __shared__ float s_cf[3][32];
    __shared__ double s_c[3][32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    DvcWarp& W = reinterpret_cast<DvcWarp*>(dvc_smem)[wl];
    unsigned char* own8 = reinterpret_cast<unsigned char*>(W.own);
    auto own_at = [&](int k) -> unsigned char& { return own8[((k >> 2) * 32 + lane) * 4 + (k & 3)]; };
    for (int c = threadIdx.x; c < a.nc; c += blockDim.x)
        s_cell[c] = (uint32_t)(c % a.nx) | (uint32_t)((c / a.nx) % a.ny) << 8 | (uint32_t)(c / (a.nx * a.ny)) << 16;
    for (int t = threadIdx.x; t < 96; t += blockDim.x) {
        s_c[t / 32][t % 32] = a.cen[t / 32][t % 32];
        s_cf[t / 32][t % 32] = (float)a.cen[t / 32][t % 32];
    }
    __syncthreads();
    // this lane's word of the grid masks
    uint32_t valid = 0, xlo = 0, xhi = 0, ylo = 0, yhi = 0;
    for (int k = 0; k < 32; ++k) {
        const int c = 32 * lane + k;
        if (c >= a.nc) continue;
        const int x = c % a.nx, y = (c / a.nx) % a.ny;
        valid |= 1u << k;
        if (x == 0) xlo |= 1u << k;
        if (x == a.nx - 1) xhi |= 1u << k;
        if (y == 0) ylo |= 1u << k;
        if (y == a.ny - 1) yhi |= 1u << k;
    }
    const int sy = a.nx, sz = a.nx * a.ny;
    auto dilate = [&](uint32_t s) {
        uint32_t r = (shl_set(s, 1, lane) & ~xlo) | (shr_set(s, 1, lane) & ~xhi);
        r |= (shl_set(s, sy, lane) & ~ylo) | (shr_set(s, sy, lane) & ~yhi);
        if (a.dim == 3) r |= shl_set(s, sz, lane) | shr_set(s, sz, lane);
        return r & valid;
    };
    // this lane's word of the set of cells point p holds
    auto cells_of = [&](int p) {
        const uint32_t p4 = (uint32_t)p * 0x01010101u;
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t eq = __vcmpeq4(W.own[j * 32 + lane], p4) & 0x08040201u;   // one bit per equal byte
            m |= ((eq | eq >> 8 | eq >> 16 | eq >> 24) & 15u) << (4 * j);
        }
        return m;
    };
    // p takes c from o when |p - c| < |o - c|.  FP32, with every coordinate in [-1, 1] rounded to 2^-24: a
    // sum of four is within 2^-20 of its value, a difference within 2^-22, so a product (factors up to 4 and
    // 2) within 1.5 2^-19 and the sum of three, with its own roundings, within 2^-16 of the FP64 value.
    constexpr float kClear = 1.0f / 32768.0f;
    const int64_t warps = (int64_t)gridDim.x * kDvcFast;
    for (int64_t e = (int64_t)blockIdx.x * kDvcFast + wl; e < a.ne; e += warps) {
        const uint32_t beg = a.offsets[e];
        const int np = (int)(a.offsets[e + 1] - beg);
        if (np > kDvcCap) {
            if (lane == 0) atomicAdd(&a.err[1], 1u);
            continue;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) W.own[j * 32 + lane] = 0xffffffffu;
        // the cell of every point (lane j: points j and j + 32), then the claims in point order
        int cell[2] = {0, 0};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int p = lane + 32 * q;
            if (p >= np) continue;
            int idx[3] = {0, 0, 0};
            const int n3[3] = {a.nx, a.ny, a.nz};
            for (int d = 0; d < a.dim; ++d) {
                const double x = a.sxi[(int64_t)d * a.nslots + beg + p];
                W.px[d][p] = (float)x;
                idx[d] = (int)__ddiv_rn(__dadd_rn(x, 1.0), a.h[d]);
                if (idx[d] == n3[d]) idx[d]--;
                // mapped points lie in [-1, 1], where this changes nothing; it keeps any other
                // value inside the grid
                idx[d] = min(max(idx[d], 0), n3[d] - 1);
            }
            cell[q] = idx[0] + a.nx * (idx[1] + a.ny * idx[2]);
        }
        __syncwarp();
        for (int p = 0; p < np; ++p) {
            const int c = __shfl_sync(0xffffffffu, p < 32 ? cell[0] : cell[1], p & 31);
            const bool here = lane == (c >> 5);
            if (here) own_at(c & 31) = (unsigned char)p;
            W.set[p * kDvcPitch + lane] = dilate(here ? 1u << (c & 31) : 0u);
        }
        __syncwarp();
        // growth passes
        const int64_t cap = (int64_t)a.nc * np + 2;
        int64_t pass = 0;
        bool taken = np > 0;
        while (taken) {
            if (++pass > cap) {
                if (lane == 0) atomicAdd(&a.err[0], 1u);
                break;
            }
            taken = false;
            for (int p = 0; p < np; ++p) {
                uint32_t b = W.set[p * kDvcPitch + lane];   // (a lane reads and writes its own word only)
                if (!__any_sync(0xffffffffu, b != 0)) continue;
                const float xp = W.px[0][p], yp = W.px[1][p], zp = a.dim == 3 ? W.px[2][p] : 0.f;
                uint32_t got = 0;
                while (b) {
                    const int k = __ffs(b) - 1;
                    b &= b - 1;
                    const int o = own_at(k);
                    bool take = o == 255;
                    if (!take && o != p) {
                        const uint32_t ci = s_cell[32 * lane + k];
                        const float cx = s_cf[0][ci & 255], cy = s_cf[1][(ci >> 8) & 255];
                        const float xo = W.px[0][o], yo = W.px[1][o];
                        float t = (xo + xp - 2.f * cx) * (xo - xp);
                        t = fmaf(yo + yp - 2.f * cy, yo - yp, t);
                        if (a.dim == 3) {
                            const float cz = s_cf[2][ci >> 16], zo = W.px[2][o];
                            t = fmaf(zo + zp - 2.f * cz, zo - zp, t);
                        }
                        take = t > 0.f;
                        if (!(fabsf(t) > kClear)) {
                            const double c0[3] = {s_c[0][ci & 255], s_c[1][(ci >> 8) & 255], s_c[2][(ci >> 16) & 31]};
                            double vo[3] = {0.0, 0.0, 0.0}, vp[3] = {0.0, 0.0, 0.0};
                            for (int d = 0; d < a.dim; ++d) {
                                vo[d] = a.sxi[(int64_t)d * a.nslots + beg + o];
                                vp[d] = a.sxi[(int64_t)d * a.nslots + beg + p];
                            }
                            take = dvc_contest(a.dim, c0, vo, vp) > 0.0;
                        }
                    }
                    if (take) {
                        own_at(k) = (unsigned char)p;
                        got |= 1u << k;
                    }
                }
                const bool any = __any_sync(0xffffffffu, got != 0);
                taken = taken || any;
                W.set[p * kDvcPitch + lane] = any ? dilate(got) & ~cells_of(p) : 0u;
            }
        }
        // centroids and weights: lane j walks the cells of point j in index order
        for (int p = 0; p < np; ++p) W.set[p * kDvcPitch + lane] = cells_of(p);
        __syncwarp();
        for (int p = lane; p < np; p += 32) {
            const uint32_t* words = W.set + p * kDvcPitch;
            double s[3] = {0.0, 0.0, 0.0};
            int cnt = 0, w = 0;
            uint32_t m = words[0];
            while (true) {
                while (m == 0 && w < 31) m = words[++w];
                if (m == 0) break;
                const uint32_t ci = s_cell[32 * w + __ffs(m) - 1];
                m &= m - 1;
                s[0] = __dadd_rn(s[0], s_c[0][ci & 255]);
                s[1] = __dadd_rn(s[1], s_c[1][(ci >> 8) & 255]);
                if (a.dim == 3) s[2] = __dadd_rn(s[2], s_c[2][ci >> 16]);
                ++cnt;
            }
            a.ow[beg + p] = __dmul_rn((double)cnt, a.da);
            for (int d = 0; d < a.dim; ++d)
                a.oxi[(int64_t)d * a.nslots + beg + p] = cnt != 0 ? __ddiv_rn(s[d], (double)cnt) : 0.0;
        }
    }
}

// The elements with more than kDvcCap points
__global__ void __launch_bounds__(32 * kDvcWarps) k_dvc_large(const __grid_constant__ DvcArgs a) {
    __shared__ int owner_s[kDvcWarps][1024];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    int* own = owner_s[wl];
    const int64_t warps = (int64_t)gridDim.x * kDvcWarps;
    // this lane's word of the grid masks
    uint32_t valid = 0, xlo = 0, xhi = 0, ylo = 0, yhi = 0;
    for (int k = 0; k < 32; ++k) {
        const int c = 32 * lane + k;
        if (c >= a.nc) continue;
        const int x = c % a.nx, y = (c / a.nx) % a.ny;
        valid |= 1u << k;
        if (x == 0) xlo |= 1u << k;
        if (x == a.nx - 1) xhi |= 1u << k;
        if (y == 0) ylo |= 1u << k;
        if (y == a.ny - 1) yhi |= 1u << k;
    }
    const int sy = a.nx, sz = a.nx * a.ny;
    auto dilate = [&](uint32_t s) {
        uint32_t r = (shl_set(s, 1, lane) & ~xlo) | (shr_set(s, 1, lane) & ~xhi);
        r |= (shl_set(s, sy, lane) & ~ylo) | (shr_set(s, sy, lane) & ~yhi);
        if (a.dim == 3) r |= shl_set(s, sz, lane) | shr_set(s, sz, lane);
        return r & valid;
    };
    for (int64_t e = (int64_t)blockIdx.x * kDvcWarps + wl; e < a.ne; e += warps) {
        const uint32_t beg = a.offsets[e];
        const int np = (int)(a.offsets[e + 1] - beg);
        if (np <= kDvcCap) continue;
        for (int k = 0; k < 32; ++k) own[k * 32 + lane] = -1;
        __syncwarp();
        // placement, in point order; the boundary of a point is the face neighbours of its cell
        for (int p = 0; p < np; ++p) {
            int idx[3] = {0, 0, 0};
            const int n3[3] = {a.nx, a.ny, a.nz};
            for (int d = 0; d < a.dim; ++d) {
                const double x = a.sxi[(int64_t)d * a.nslots + beg + p];
                idx[d] = (int)__ddiv_rn(__dadd_rn(x, 1.0), a.h[d]);
                if (idx[d] == n3[d]) idx[d]--;
                // mapped points lie in [-1, 1], where this changes nothing; it keeps any other
                // value inside the grid
                idx[d] = min(max(idx[d], 0), n3[d] - 1);
            }
            const int c = idx[0] + a.nx * (idx[1] + a.ny * idx[2]);
            if (lane == (c >> 5)) own[(c & 31) * 32 + lane] = p;
            const uint32_t one = lane == (c >> 5) ? 1u << (c & 31) : 0u;
            a.bnd[(int64_t)(beg + p) * 32 + lane] = dilate(one);
            __syncwarp();
        }
        // growth passes
        const int64_t cap = (int64_t)a.nc * np + 2;
        int64_t pass = 0;
        bool taken = np > 0;
        while (taken) {
            if (++pass > cap) {
                if (lane == 0) atomicAdd(&a.err[0], 1u);
                break;
            }
            int total = 0;
            for (int p = 0; p < np; ++p) {
                uint32_t* bw = a.bnd + (int64_t)(beg + p) * 32;
                uint32_t b = bw[lane];
                double xp[3] = {0.0, 0.0, 0.0};
                for (int d = 0; d < a.dim; ++d) xp[d] = a.sxi[(int64_t)d * a.nslots + beg + p];
                uint32_t got = 0;
                while (b) {
                    const int k = __ffs(b) - 1;
                    b &= b - 1;
                    const int c = 32 * lane + k;
                    const int o = own[k * 32 + lane];
                    bool take = o == -1;
                    if (!take && o != p) {
                        const double c0[3] = {a.cen[0][c % a.nx], a.cen[1][(c / a.nx) % a.ny],
                                              a.dim == 3 ? a.cen[2][c / (a.nx * a.ny)] : 0.0};
                        double xo[3] = {0.0, 0.0, 0.0};
                        for (int d = 0; d < a.dim; ++d) xo[d] = a.sxi[(int64_t)d * a.nslots + beg + o];
                        take = dvc_contest(a.dim, c0, xo, xp) > 0.0;
                    }
                    if (take) {
                        own[k * 32 + lane] = p;
                        got |= 1u << k;
                    }
                }
                __syncwarp();
                total += __popc(got);
                uint32_t mine = 0;
                for (int k = 0; k < 32; ++k) mine |= (own[k * 32 + lane] == p ? 1u : 0u) << k;
                bw[lane] = dilate(got) & ~mine;
                __syncwarp();
            }
            taken = __any_sync(0xffffffffu, total != 0);
        }
        // centroids and weights: lane j accumulates point j over the cells in index order
        for (int p0 = 0; p0 < np; p0 += 32) {
            const int p = p0 + lane;
            double s[3] = {0.0, 0.0, 0.0};
            int cnt = 0;
            int x = 0, y = 0, z = 0;
            for (int c = 0; c < a.nc; ++c) {
                if (own[(c & 31) * 32 + (c >> 5)] == p) {
                    s[0] = __dadd_rn(s[0], a.cen[0][x]);
                    s[1] = __dadd_rn(s[1], a.cen[1][y]);
                    if (a.dim == 3) s[2] = __dadd_rn(s[2], a.cen[2][z]);
                    ++cnt;
                }
                if (++x == a.nx) {
                    x = 0;
                    if (++y == a.ny) {
                        y = 0;
                        ++z;
                    }
                }
            }
            if (p < np) {
                a.ow[beg + p] = __dmul_rn((double)cnt, a.da);
                for (int d = 0; d < a.dim; ++d)
                    a.oxi[(int64_t)d * a.nslots + beg + p] = cnt != 0 ? __ddiv_rn(s[d], (double)cnt) : 0.0;
            }
        }
        __syncwarp();
    }
}

// the constant weights 2^dim / count of the element (ConstantWeights.c:180-189)
__global__ void k_const_weights(int64_t ne, int dim, const uint32_t* __restrict__ offsets, double* __restrict__ w) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const uint32_t beg = offsets[e], end = offsets[e + 1];
    const double v = (dim == 3 ? 8.0 : 4.0) / (double)(end - beg);
    for (uint32_t s = beg; s < end; ++s) w[s] = v;
}

}  // namespace

void weights_set(Context& c, int kind, const int32_t res[3]) {
    UWG_REQUIRE(kind == UWGPU_WEIGHTS_CONSTANT || kind == UWGPU_WEIGHTS_DVC, UWGPU_ERR_ARGUMENT,
                "weights kind must be UWGPU_WEIGHTS_CONSTANT or UWGPU_WEIGHTS_DVC");
    if (kind == UWGPU_WEIGHTS_DVC) {
        UWG_REQUIRE(res != nullptr, UWGPU_ERR_ARGUMENT, "DVC weights need a resolution");
        const int dim = c.has_mesh ? c.mesh.dim : 3;
        int64_t nc = 1;
        for (int d = 0; d < dim; ++d) {
            UWG_REQUIRE(res[d] >= 1 && res[d] <= 32, UWGPU_ERR_ARGUMENT, "DVC resolution must be 1..32 per axis");
            nc *= res[d];
        }
        UWG_REQUIRE(nc <= 1024, UWGPU_ERR_ARGUMENT, "DVC grid limited to 1024 cells per element");
        for (int d = 0; d < 3; ++d) c.dvc_res[d] = d < dim ? res[d] : 1;
    }
    c.weights_kind = kind;
    c.assembled = false;
    c.operator_built = false;
}

// The integration points of the next assembly: with DVC weights, the Voronoi centroids and
// volumes of the mapped points (c.dvc_xi, c.dvc_w); returns the local coordinates to assemble
// from and the per-slot weights (null: constant weights).
void integration_points(Context& c, const double** xi, const double** w) {
    const MeshDesc& m = c.mesh;
    if (c.weights_kind != UWGPU_WEIGHTS_DVC) {
        *xi = c.sxi.p;
        *w = nullptr;
        return;
    }
    const int dim = m.dim;
    int64_t nc = 1;
    for (int d = 0; d < dim; ++d) nc *= c.dvc_res[d];
    UWG_REQUIRE(nc <= 1024, UWGPU_ERR_ARGUMENT, "DVC grid limited to 1024 cells per element");
    const size_t ns = (size_t)(c.np > 0 ? c.np : 1);
    c.dvc_xi.ensure((size_t)dim * ns);
    c.dvc_w.ensure(ns);
    c.err_count.ensure(2);
    UWG_CUDA(cudaMemsetAsync(c.err_count.p, 0, 2 * sizeof(uint32_t), c.stream));
    DvcArgs a;
    std::memset(&a, 0, sizeof(a));
    a.dim = dim;
    a.nx = c.dvc_res[0];
    a.ny = c.dvc_res[1];
    a.nz = dim == 3 ? c.dvc_res[2] : 1;
    a.nc = (int)nc;
    const int n3[3] = {a.nx, a.ny, a.nz};
    for (int d = 0; d < 3; ++d) {
        // _DVCWeights_ConstructGrid: h = (1 - (-1)) / res, centre = -1 - h/2, then + h per cell
        const double h = 2.0 / n3[d];
        a.h[d] = h;
        double x = -1.0 - h / 2.0;
        for (int i = 0; i < n3[d] && i < 32; ++i) {
            x = x + h;
            a.cen[d][i] = x;
        }
    }
    a.da = dim == 3 ? a.h[0] * a.h[1] * a.h[2] : a.h[0] * a.h[1];
    a.ne = m.ne;
    a.nslots = c.np;
    a.offsets = c.offsets.p;
    a.sxi = c.sxi.p;
    a.oxi = c.dvc_xi.p;
    a.ow = c.dvc_w.p;
    a.bnd = nullptr;
    a.err = c.err_count.p;
    uint32_t err[2] = {0, 0};
    auto read_err = [&]() {
        UWG_CUDA(cudaMemcpyAsync(c.host_scalars, c.err_count.p, sizeof(err), cudaMemcpyDeviceToHost, c.stream));
        UWG_CUDA(cudaStreamSynchronize(c.stream));
        std::memcpy(err, c.host_scalars, sizeof(err));
    };
    if (m.ne > 0 && c.np > 0) {
        int sms = 0;
        UWG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
        {
            LaunchScope ls(c, UWGPU_KERNEL_ASSEMBLY);
            const size_t smem = kDvcFast * sizeof(DvcWarp);
            UWG_CUDA(cudaFuncSetAttribute(k_dvc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            const int64_t want = (m.ne + kDvcFast - 1) / kDvcFast;
            k_dvc<<<(unsigned)std::min<int64_t>(want, (int64_t)sms * 16), 32 * kDvcFast, smem, c.stream>>>(a);
            note_work(c, UWGPU_KERNEL_ASSEMBLY, (double)c.np * (dim * 16.0 + 8.0), (double)c.np * nc * 4.0);
        }
        check_launch("k_dvc");
        read_err();
        if (err[1] && !err[0]) {   // elements with more points than its shared memory holds
            c.dvc_bnd.ensure(32 * ns);
            a.bnd = c.dvc_bnd.p;
            LaunchScope ls(c, UWGPU_KERNEL_ASSEMBLY);
            const int64_t want = (m.ne + kDvcWarps - 1) / kDvcWarps;
            k_dvc_large<<<(unsigned)std::min<int64_t>(want, (int64_t)sms * 16), 32 * kDvcWarps, 0, c.stream>>>(a);
            check_launch("k_dvc_large");
            read_err();
        }
    }
    if (err[0]) throw Error(UWGPU_ERR_NOT_CONVERGED, "DVC weights: region growth did not settle");
    *xi = c.dvc_xi.p;
    *w = c.dvc_w.p;
}

// the local coordinates ([slot][3] on the host) and weights the last assembly integrated with
void integration_points_download(Context& c, double* xi, double* w) {
    UWG_REQUIRE(c.assembled, UWGPU_ERR_STATE, "nothing assembled");
    const int dim = c.mesh.dim;
    const size_t N = (size_t)c.np;
    if (N == 0) return;
    const double* src = c.weights_kind == UWGPU_WEIGHTS_DVC ? c.dvc_xi.p : c.sxi.p;
    if (xi) {
        vector_to_host<double>(c, (int64_t)N, dim, 3, src, xi);
        UWG_CUDA(cudaStreamSynchronize(c.stream));
    }
    if (w) {
        if (c.weights_kind == UWGPU_WEIGHTS_DVC) {
            UWG_CUDA(cudaMemcpyAsync(w, c.dvc_w.p, N * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
        } else {
            DArray<double> tw;
            tw.ensure(N);
            {
                LaunchScope ls(c, -1);
                k_const_weights<<<blocks_for(c.mesh.ne, 256), 256, 0, c.stream>>>(c.mesh.ne, dim, c.offsets.p, tw.p);
            }
            check_launch("k_const_weights");
            UWG_CUDA(cudaMemcpyAsync(w, tw.p, N * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
            UWG_CUDA(cudaStreamSynchronize(c.stream));
        }
        UWG_CUDA(cudaStreamSynchronize(c.stream));
    }
}

}  // namespace uwg
