// Node-block stencil: grid description and indexing shared by the operator kernels (operator.cu) and the
// one-launch cycle of small multigrid levels (cycle.cu).
#pragma once

#include "internal.cuh"

namespace uwg {

struct Grid {
    int dim;
    int64_t nx, ny, nz;  // nodes per axis
    int64_t nn;
    int ex, ey, ez;      // elements per axis
};

inline Grid grid_of(const MeshDesc& m) {
    Grid g;
    g.dim = m.dim;
    g.nx = m.nnx;
    g.ny = m.nny;
    g.nz = m.nnz;
    g.nn = m.nn;
    g.ex = m.nel[0];
    g.ey = m.nel[1];
    g.ez = m.dim == 3 ? m.nel[2] : 1;
    return g;
}

template <int DIM>
__host__ __device__ constexpr int nblocks() { return DIM == 3 ? 27 : 9; }

// Neighbour offsets of node (i, j, k) per axis, 0 towards a missing neighbour.  Every stencil block
// towards a neighbour outside the mesh is stored as zero, so a row reads the node itself there
// and all loads of a row are unconditional (they can all be in flight at once).
struct NbrOffsets {
    int64_t dx[3], dy[3], dz[3];
};

template <int DIM>
__device__ __forceinline__ NbrOffsets nbr_offsets(const Grid& g, int64_t i, int64_t j, int64_t k) {
    NbrOffsets o;
    o.dx[0] = i > 0 ? -1 : 0;
    o.dx[1] = 0;
    o.dx[2] = i + 1 < g.nx ? 1 : 0;
    o.dy[0] = j > 0 ? -g.nx : 0;
    o.dy[1] = 0;
    o.dy[2] = j + 1 < g.ny ? g.nx : 0;
    o.dz[0] = DIM == 3 && k > 0 ? -g.nx * g.ny : 0;
    o.dz[1] = 0;
    o.dz[2] = DIM == 3 && k + 1 < g.nz ? g.nx * g.ny : 0;
    return o;
}

// (i, j, k) of node n with 32-bit division (node counts stay below 2^32, checked on the host)
template <int DIM>
__device__ __forceinline__ void node_ijk(const Grid& g, int64_t n, int64_t& i, int64_t& j, int64_t& k) {
    const unsigned un = (unsigned)n, nx = (unsigned)g.nx, ny = (unsigned)g.ny;
    const unsigned q = un / nx;
    i = un - q * nx;
    j = DIM == 3 ? q % ny : q;
    k = DIM == 3 ? q / ny : 0;
}

// ------------------------------------------------------------------------------------------
// Split rows.  A warp works on 32 nodes (lanes), one of their DIM rows and one third of the row's
// neighbours (a z plane of the stencil in 3D, a y row in 2D), so that all loads of a row third are in
// flight at once and a row costs one memory latency instead of a chain of them.  A group of 3 DIM
// warps covers 32 nodes; the partial sums meet in shared memory.
// ------------------------------------------------------------------------------------------
constexpr int kSplitThreads = 576;   // 18 warps: 2 groups of 9 in 3D, 3 groups of 6 in 2D

template <int DIM>
struct Split {
    static constexpr int kGroupWarps = 3 * DIM;
    static constexpr int kGroups = kSplitThreads / 32 / kGroupWarps;
    static constexpr int kNodes = 32 * kGroups;   // nodes a block handles at once
};

// Third s of row r of node n: sum over its neighbours of A[q][r][c][n] x[c][m(q)].  x is read past
// L1: other SMs write it between the phases of one launch.
template <int DIM, typename T>
__device__ __forceinline__ T row_part(const Grid& g, int64_t n, int64_t i, int64_t j, int64_t k, int r, int s,
                                      const T* __restrict__ A, const T* x) {
    constexpr int NQ = DIM == 3 ? 9 : 3;
    const NbrOffsets o = nbr_offsets<DIM>(g, i, j, k);
    const int64_t po = DIM == 3 ? (s == 0 ? o.dz[0] : s == 2 ? o.dz[2] : 0) : (s == 0 ? o.dy[0] : s == 2 ? o.dy[2] : 0);
    const T* Ar = A + ((int64_t)(s * NQ * DIM + r) * DIM) * g.nn + n;
    T a[NQ * DIM], xv[NQ * DIM];
#pragma unroll
    for (int t = 0; t < NQ; ++t) {
        const int64_t m = n + po + o.dx[t % 3] + (DIM == 3 ? o.dy[(t / 3) % 3] : 0);
#pragma unroll
        for (int cc = 0; cc < DIM; ++cc) {
            a[t * DIM + cc] = __ldg(Ar + (int64_t)(t * DIM * DIM + cc) * g.nn);
            xv[t * DIM + cc] = __ldcg(x + (int64_t)cc * g.nn + m);
        }
    }
    T out = (T)0;
#pragma unroll
    for (int t = 0; t < NQ * DIM; ++t) out = fma(a[t], xv[t], out);
    return out;
}

// One colour of a block Gauss-Seidel sweep by blocks cta of ncta: x_n += Dinv_n (b_n - (A x)_n) on
// the nodes of parity `col`, which share no stencil entry.  sres: two buffers of kSplitThreads; the
// caller separates the colours by a barrier over all blocks.
template <int DIM, typename T>
__device__ __forceinline__ void gs_colour(const Grid& g, const T* __restrict__ A, const T* __restrict__ Dinv,
                                          const T* b, T* x, int col, int cta, int ncta, T* sres) {
    typedef Split<DIM> S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = warp / S::kGroupWarps, wi = warp % S::kGroupWarps, r = wi / 3, s = wi % 3;
    const int px = col & 1, py = (col >> 1) & 1, pz = (col >> 2) & 1;
    const int64_t cx = (g.nx - px + 1) / 2, cy = (g.ny - py + 1) / 2;
    const int64_t cnt = cx * cy * (DIM == 3 ? (g.nz - pz + 1) / 2 : 1);
    int buf = 0;
    for (int64_t base = (int64_t)cta * S::kNodes; base < cnt; base += (int64_t)ncta * S::kNodes) {
        const int64_t t = base + grp * 32 + lane;
        const bool act = t < cnt;
        int64_t n = 0;
        T part = (T)0, bv[DIM], dv[DIM], v = (T)0;
        if (act) {
            const unsigned ut = (unsigned)t, q = ut / (unsigned)cx, q2 = DIM == 3 ? q / (unsigned)cy : 0u;
            const int64_t i = 2 * (int64_t)(ut - q * (unsigned)cx) + px;
            const int64_t j = 2 * (int64_t)(DIM == 3 ? q - q2 * (unsigned)cy : q) + py;
            const int64_t k = DIM == 3 ? 2 * (int64_t)q2 + pz : 0;
            n = i + g.nx * (j + g.ny * k);
            if (s == 0) {
                v = __ldcg(x + (int64_t)r * g.nn + n);
#pragma unroll
                for (int cc = 0; cc < DIM; ++cc) {
                    bv[cc] = __ldcg(b + (int64_t)cc * g.nn + n);
                    dv[cc] = __ldg(Dinv + (int64_t)(r * DIM + cc) * g.nn + n);
                }
            }
            part = row_part<DIM, T>(g, n, i, j, k, r, s, A, x);
        }
        T* sb = sres + buf * kSplitThreads;
        buf ^= 1;   // the barrier of the next round separates this round's reads from the next but one's writes
        sb[threadIdx.x] = part;
        __syncthreads();
        if (act && s == 0) {
#pragma unroll
            for (int cc = 0; cc < DIM; ++cc) {
                const T* p = sb + (grp * S::kGroupWarps + cc * 3) * 32 + lane;
                v = fma(dv[cc], bv[cc] - ((p[0] + p[32]) + p[64]), v);
            }
            x[(int64_t)r * g.nn + n] = v;
        }
    }
}

// Colours of `sweeps` symmetric sweeps in order (ascending, then descending).  A colour that follows
// itself is left out: its nodes were just solved exactly and nothing they depend on has changed, so
// relaxing them again adds a zero correction.
template <int DIM>
__host__ __device__ constexpr int gs_steps(int sweeps) {
    return sweeps <= 0 ? 0 : 1 + sweeps * 2 * ((1 << DIM) - 1);
}
template <int DIM>
__host__ __device__ constexpr int gs_step_colour(int step) {
    constexpr int P = (1 << DIM) - 1;   // 0 .. P .. 0 .. P ..: a triangle wave
    const int q = step % (2 * P);
    return q <= P ? q : 2 * P - q;
}

}  // namespace uwg
