// Small multigrid levels and small velocity solves in one launch.
//
// On a small level a kernel of the V-cycle runs for 2 to 4 us, and the colour smoother's grid barrier
// (4,600 cycles with cooperative groups) costs more than the colour it separates, so a cycle over small
// levels was bound by launches and barriers.  Here one cooperative launch with one block per SM runs every
// phase of the cycle from a given level down to the coarsest and back (smoothing, residual, restriction,
// coarse solve, prolongation).  When even the finest level is small, it goes on with the rest of a flexible
// GMRES iteration: w = A z, classical Gram-Schmidt with one re-orthogonalisation, and the next basis
// vector; the host reads the column of H once per iteration.
//
// A phase costs one pass of its data through L2 and one barrier (3,100 cycles for a store, the barrier and
// a dependent load, whether 16 or 152 blocks take part; 2,200 inside a 16-block cluster).  An FP64 FMA
// occupies a scheduler for 64 cycles per warp on this part, so a cluster's 16 SMs were bound by the FP64
// pipe (a 17^3 level: 4 us a colour) and the whole chip is the better place.  Per phase, the nodes are
// split evenly over the blocks, a row of a node over three threads (27 instead of 81 dependent FMAs), and
// the work of a block is packed into as few warps as hold it.  What a smoothing call does not change
// (stencil, inverse diagonal, right-hand side) is fetched between arriving at a barrier and waiting on it.
//
// In 2D the colours of a Gauss-Seidel call, most of a cycle's phases, are not separated by barriers: every
// value is kept beside a tag that names the step that formed it, in one word that is read and written whole,
// and a row polls its neighbours until each carries the tag of its colour's last step.  A node cannot be
// relaxed again before its neighbours have used the value (its next relaxation waits for theirs), so the
// colours follow each other through the data.  Per V-cycle iteration: 65^2 237 -> 196 us, 129^2 255 -> 210,
// 257^2 393 -> 349.  In 3D a thread polls 27 words instead of 6 and the barrier is the faster (17^3 456 us
// against 525).
//
// Vectors written during the launch are read past L1 (__ldcg).  The arithmetic is that of the per-kernel
// path (operator.cu, solver.cu) up to the order of sums.  A lane adds up to 59 products of a Gram-Schmidt sum
// (40,000 nodes) where that path has one per thread, FP64 from the warps on: FP32 products are added in pairs
// (longsum.cuh), which takes an iteration of a 33^3 level from 199.5 to 201.2 us.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "cycle.cuh"
#include "longsum.cuh"
#include "stencil.cuh"

namespace uwg {

namespace {

constexpr int kCyThreads = 256;
constexpr int kCyKrylovBlocks = 64;     // blocks of the Gram-Schmidt part (each adds up all partial sums)
constexpr int kCyWait = 1 << 22;        // polls of a barrier before the launch gives up
constexpr int kCyPolls = 1 << 20;       // polls of a row's neighbours
constexpr int kCySweeps = 256;          // most smoothing sweeps per call
// Levels (nodes) up to which the cycle runs here, per smoother, measured per V-cycle iteration of whole
// velocity solves (us, all levels as separate kernels / this level and below here): colour sweeps, which
// alternate with barriers, 2D 65^2 461 / 196, 129^2 490 / 210, 257^2 547 / 349; 3D 17^3 1167 / 456, 33^3
// 1408 / 781, 41^3 1986 / 1254 (81,000 nodes and more were not tried, the kernels win at 65^3: 1014
// against 585 with Chebyshev).  Chebyshev in mixed precision: 17^3 226 / 117, 33^3 289 / 215 with the whole
// iteration here; as levels below a 65^3 mesh 17^3 and less gain (585 / 577), 33^3 does not (590).
constexpr int64_t kCyNodesColour = 80000, kCyNodesCheb = 6000, kCyNodesWhole = 40000;

// A value and the tag of the step that formed it, in one naturally aligned word of 16 or 8 bytes
template <typename T>
struct alignas(2 * sizeof(T)) Tagged {
    T v;
    uint32_t tag;
};
__device__ __forceinline__ Tagged<double> load_tagged(const Tagged<double>* p) {
    uint64_t a, b;
    asm volatile("{ .reg .b128 q; ld.relaxed.gpu.global.b128 q, [%2]; mov.b128 {%0, %1}, q; }" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    return Tagged<double>{__longlong_as_double((long long)a), (uint32_t)b};
}
__device__ __forceinline__ void store_tagged(Tagged<double>* p, double v, uint32_t tag) {
    asm volatile("{ .reg .b128 q; mov.b128 q, {%1, %2}; st.relaxed.gpu.global.b128 [%0], q; }" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((uint64_t)tag)
                 : "memory");
}
__device__ __forceinline__ Tagged<float> load_tagged(const Tagged<float>* p) {
    uint64_t a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return Tagged<float>{__uint_as_float((uint32_t)a), (uint32_t)(a >> 32)};
}
__device__ __forceinline__ void store_tagged(Tagged<float>* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((uint64_t)__float_as_uint(v) | (uint64_t)tag << 32) : "memory");
}

// Last step before `step` of the triangle wave of colours (gs_step_colour) that relaxed colour c; -1: none
template <int DIM>
__host__ __device__ constexpr int last_step(int step, int c) {
    constexpr int P = (1 << DIM) - 1;
    const int q = step % (2 * P), base = step - q;
    const int down = c == 0 ? 2 * P : 2 * P - c;   // the colour's descending place in a period (0: the next period)
    if (down < q) return base + down;
    if (c < q) return base + c;
    return base == 0 ? -1 : base - 2 * P + (c == 0 ? 0 : 2 * P - c);
}
constexpr bool last_step_ok() {
    int last[4] = {-1, -1, -1, -1};
    for (int step = 0; step < gs_steps<2>(3); ++step) {
        for (int c = 0; c < 4; ++c)
            if (last_step<2>(step, c) != last[c]) return false;
        last[gs_step_colour<2>(step)] = step;
    }
    return true;
}
static_assert(last_step_ok(), "last_step and gs_step_colour disagree");

template <typename T>
struct CyLevel {
    Grid g;
    const T* A;
    const uint32_t* A16;   // FP16 row-scaled copy (mixed form), or null
    const float* S16;
    const T* Dinv;
    T *b, *x, *r, *t;      // right-hand side, iterate, residual or Chebyshev direction, alternate iterate
    Tagged<T>* xt;         // 2D: the iterate with the tags of a Gauss-Seidel call
    const uint8_t* fixed;
    T c1[kCyMaxDegree], c2[kCyMaxDegree];   // Chebyshev recurrence (k_cheb_step)
};

template <typename T>
struct CyArgs {
    CyLevel<T> L[kCyMaxLevels];
    int nlev, cheb, down, up;
    const double* Cinv;
    int64_t ncoarse;
    uint32_t* bar;         // [0] this launch's barrier count, [1] the next launch's (cleared here), [2] error
    int which;             // which of the two counts this launch uses
    uint32_t tag;          // first tag of this launch (2D)
    int64_t n;             // unknowns of the finest level
    // Krylov part (V null: the cycle alone): vectors V_j of n entries, j <= k
    const T* V;
    T* vnext;
    T* w;
    double* part;          // [3][kCyPass][kCyKrylovBlocks]
    int k;
    double* out;           // host memory: H column of the two passes at 0 and kCyPass, ||w||^2 at 2 kCyPass
};

// Barrier over the grid, split in two: arrive (all of the block's earlier stores are released) and wait.
// A wait that runs out ends all later waits of the block and reports an error.
struct GridBarrier {
    uint32_t* count;
    uint32_t* err;
    uint32_t target = 0;
    bool ok = true, pending = false;   // pending: arrived and not yet waited (the same in every thread)
    __device__ __forceinline__ void arrive() {
        __syncthreads();
        pending = true;
        target += gridDim.x;
        if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    }
    __device__ __forceinline__ void wait() {
        if (!pending) return;
        pending = false;
        if (threadIdx.x == 0 && ok) {
            uint32_t cur;
            int polls = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(count) : "memory");
            } while (cur < target && ++polls < kCyWait);
            if (cur < target) {
                ok = false;
                atomicOr(err, 1u);
            }
        }
        __syncthreads();
    }
    __device__ __forceinline__ void sync() {
        arrive();
        wait();
    }
};

// One third (a z plane of the stencil in 3D, a y row in 2D) of a row: its stencil entries, and their
// product with x.  NQ neighbours of DIM components; the FP16 form holds two neighbours per word, five
// words per third in 3D (ten neighbours) and two in 2D.
template <int DIM, typename T, bool HALF>
struct RowThird {
    static constexpr int NB = nblocks<DIM>(), NP = (NB + 1) / 2, PB = (NP + 2) / 3, NQ = NB / 3;
    T a[HALF ? 1 : NQ * DIM];
    uint32_t h[HALF ? PB * DIM : 1];
    __device__ __forceinline__ void load(const CyLevel<T>& L, int n, int r, int s) {
        const int nn = (int)L.g.nn;
        if constexpr (HALF) {
            const uint32_t* p = L.A16 + (s * PB * DIM + r) * DIM * nn + n;
#pragma unroll
            for (int t = 0; t < PB; ++t)
#pragma unroll
                for (int cc = 0; cc < DIM; ++cc) h[t * DIM + cc] = s * PB + t < NP ? __ldg(p + (t * DIM * DIM + cc) * nn) : 0u;
        } else {
            const T* p = L.A + (s * NQ * DIM + r) * DIM * nn + n;
#pragma unroll
            for (int t = 0; t < NQ; ++t)
#pragma unroll
                for (int cc = 0; cc < DIM; ++cc) a[t * DIM + cc] = __ldg(p + (t * DIM * DIM + cc) * nn);
        }
    }
    // 2D: the product with the tagged iterate; polls until every neighbour carries its colour's last tag before
    // `step` (tag0 for the initial values; zero: those are zero and nothing is read); false when it gave up
    __device__ __forceinline__ bool dot_tagged(const CyLevel<T>& L, int n, int s, int col, int step, uint32_t tag0, bool zero,
                                               bool poll, T& out) const {
        static_assert(DIM == 2, "the tagged iterate is the 2D form");
        const Grid& g = L.g;
        const int nn = (int)g.nn, nx = (int)g.nx;
        int64_t i, j, k;
        node_ijk<DIM>(g, n, i, j, k);
        const bool in = s == 0 ? j > 0 : s == 1 || j + 1 < g.ny;   // the third (row j + s - 1) lies in the mesh
        const int row = n + (s - 1) * nx;
        uint32_t want[2];   // tag to wait for, of the neighbours in this and in the next columns; 0: nothing to read
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int last = last_step<DIM>(step, (s == 1 ? col : col ^ 2) ^ q);
            want[q] = last < 0 ? (zero ? 0u : tag0) : tag0 + 1u + (uint32_t)last;
        }
        const bool live[3] = {in && i > 0 && want[1], in && want[0], in && i + 1 < g.nx && want[1]};
        T xv[NQ * DIM];
        bool ready;
        int polls = 0;
        do {
            ready = true;
#pragma unroll
            for (int t = 0; t < NQ; ++t)
#pragma unroll
                for (int cc = 0; cc < DIM; ++cc) {
                    xv[t * DIM + cc] = (T)0;
                    if (live[t]) {
                        const Tagged<T> e = load_tagged(L.xt + cc * nn + row + t - 1);
                        xv[t * DIM + cc] = e.v;
                        ready = ready && e.tag == want[(t + 1) & 1];
                    }
                }
        } while (!ready && poll && ++polls < kCyPolls);
        out = (T)0;
#pragma unroll
        for (int t = 0; t < NQ * DIM; ++t) out = fma(a[t], xv[t], out);
        return ready;
    }
    __device__ __forceinline__ T dot(const CyLevel<T>& L, int n, int s, const T* x) const {
        const Grid& g = L.g;
        const int nn = (int)g.nn;
        int64_t i, j, k;
        node_ijk<DIM>(g, n, i, j, k);
        const int dx[3] = {i > 0 ? -1 : 0, 0, i + 1 < g.nx ? 1 : 0};
        const int dy[3] = {j > 0 ? -(int)g.nx : 0, 0, j + 1 < g.ny ? (int)g.nx : 0};
        const int pl = (int)(g.nx * g.ny);
        const int dz[3] = {DIM == 3 && k > 0 ? -pl : 0, 0, DIM == 3 && k + 1 < g.nz ? pl : 0};
        T out = (T)0;
        if constexpr (HALF) {
            auto third = [&](auto sc) {
                constexpr int S = decltype(sc)::value;
                T xv[2 * PB * DIM];
#pragma unroll
                for (int t = 0; t < PB; ++t) {
                    const int q0 = 2 * (S * PB + t), q1 = q0 + 1;
                    if (S * PB + t < NP) {
                        const int m0 = n + dx[q0 % 3] + dy[(q0 / 3) % 3] + dz[DIM == 3 ? q0 / 9 : 1];
                        const int m1 = q1 < NB ? n + dx[q1 % 3] + dy[(q1 / 3) % 3] + dz[DIM == 3 ? q1 / 9 : 1] : n;
#pragma unroll
                        for (int cc = 0; cc < DIM; ++cc) {
                            xv[2 * t * DIM + cc] = __ldcg(x + cc * nn + m0);
                            xv[(2 * t + 1) * DIM + cc] = q1 < NB ? __ldcg(x + cc * nn + m1) : (T)0;
                        }
                    }
                }
#pragma unroll
                for (int t = 0; t < PB; ++t)
                    if (S * PB + t < NP) {
#pragma unroll
                        for (int cc = 0; cc < DIM; ++cc) {
                            const uint32_t wv = h[t * DIM + cc];
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&wv));
                            out = fmaf(f.x, xv[2 * t * DIM + cc], out);
                            out = fmaf(f.y, xv[(2 * t + 1) * DIM + cc], out);
                        }
                    }
            };
            if (s == 0) third(std::integral_constant<int, 0>());
            else if (s == 1) third(std::integral_constant<int, 1>());
            else third(std::integral_constant<int, 2>());
        } else {
            const int po = n + (DIM == 3 ? (s == 0 ? dz[0] : s == 2 ? dz[2] : 0) : (s == 0 ? dy[0] : s == 2 ? dy[2] : 0));
            T xv[NQ * DIM];
#pragma unroll
            for (int t = 0; t < NQ; ++t)
#pragma unroll
                for (int cc = 0; cc < DIM; ++cc)
                    xv[t * DIM + cc] = __ldcg(x + cc * nn + po + dx[t % 3] + (DIM == 3 ? dy[(t / 3) % 3] : 0));
#pragma unroll
            for (int t = 0; t < NQ * DIM; ++t) out = fma(a[t], xv[t], out);
        }
        return out;
    }
};

// share of `count` items that this block takes: first item and how many
__device__ __forceinline__ void block_share(int count, int& first, int& mine) {
    const int per = (count + (int)gridDim.x - 1) / (int)gridDim.x;
    first = (int)blockIdx.x * per;
    mine = max(0, min(per, count - first));
}

enum { kApply = 0, kResidual = 1, kCheb = 2 };

// All nodes of a level, a block's share in rounds of kCyThreads / (3 DIM) nodes.  kApply: y = A x;
// kResidual: y = b - A x;  kCheb: z = Dinv (b - A x), d = c1 d + c2 z, y = x + d (x null: zero; first:
// d = c2 z).
template <int DIM, typename T, bool HALF, int MODE>
__device__ __forceinline__ void node_phase(const CyLevel<T>& L, const T* x, T* y, T c1, T c2, bool first, T* sres) {
    constexpr int W = 3 * DIM, ROUND = kCyThreads / W;
    const int nn = (int)L.g.nn;
    int n0, mine;
    block_share(nn, n0, mine);
    for (int base = 0; base < mine; base += ROUND) {
        const int cnt = min(ROUND, mine - base);
        const int it = threadIdx.x, combo = it / cnt, loc = it - combo * cnt, n = n0 + base + loc;
        T part = (T)0, bv[DIM], dv[DIM], sv[DIM], own = (T)0, dold = (T)0;
        const int r = combo, idx = r * nn + n;   // (the rows' sums: combo < DIM)
        if (combo < DIM) {
#pragma unroll
            for (int cc = 0; cc < DIM; ++cc) {
                if (MODE == kCheb) dv[cc] = __ldg(L.Dinv + (r * DIM + cc) * nn + n);
                if (MODE == kCheb) bv[cc] = __ldcg(L.b + cc * nn + n);
                if (HALF && MODE == kCheb) sv[cc] = (T)__ldg(L.S16 + cc * nn + n);
            }
            if (MODE == kResidual) bv[0] = __ldcg(L.b + idx);
            if (HALF && MODE == kResidual) sv[0] = (T)__ldg(L.S16 + idx);
            if (MODE == kCheb && x) own = __ldcg(x + idx);
            if (MODE == kCheb && !first) dold = __ldcg(L.r + idx);
        }
        if (x && combo < W) {
            RowThird<DIM, T, HALF> row;
            row.load(L, n, combo / 3, combo % 3);
            part = row.dot(L, n, combo % 3, x);
        }
        if (base) __syncthreads();   // the previous round's sums have been read
        if (combo < W) sres[it] = part;
        __syncthreads();
        if (combo < DIM) {
            if (MODE == kCheb) {
                T z = (T)0;
#pragma unroll
                for (int cc = 0; cc < DIM; ++cc) {
                    const T* p = sres + cc * 3 * cnt + loc;
                    T ax = (p[0] + p[cnt]) + p[2 * cnt];
                    if (HALF) ax *= sv[cc];
                    z = fma(dv[cc], bv[cc] - ax, z);
                }
                const T dn = first ? c2 * z : fma(c1, dold, c2 * z);
                L.r[idx] = dn;
                y[idx] = own + dn;
            } else {
                const T* p = sres + r * 3 * cnt + loc;
                T ax = (p[0] + p[cnt]) + p[2 * cnt];
                if (HALF && MODE == kResidual) ax *= sv[0];
                y[idx] = MODE == kResidual ? bv[0] - ax : ax;
            }
        }
    }
}

template <int DIM, typename T, bool HALF>
__global__ void __launch_bounds__(kCyThreads, 1) k_cycle(const __grid_constant__ CyArgs<T> a) {
    __shared__ T sres[2 * kCyThreads];
    __shared__ double s_h[kCyPass];
    __shared__ int s_dead;   // a poll of this block has run out: no more polling
    const int tid = threadIdx.x, gt = (int)blockIdx.x * kCyThreads + tid, gn = (int)gridDim.x * kCyThreads;
    constexpr int W = 3 * DIM, ROUND = kCyThreads / W;
    GridBarrier bar{a.bar + a.which, a.bar + 2};
    if (gt == 0) a.bar[a.which ^ 1] = 0u;   // the next launch's count
    if (tid == 0) s_dead = 0;
    __syncthreads();

    // symmetric colour Gauss-Seidel (gs_steps, gs_step_colour).  A barrier may be pending on entry, and one
    // is on exit: whoever needs the values waits.  b and the stencil do not change here.  2D: on the tagged
    // iterate, from zero or from the values stored with tag `tag`; the block's partial sums alternate between
    // two buffers, so one block barrier per round orders them.
    uint32_t tag = a.tag;
    auto smooth_gs = [&](const CyLevel<T>& L, int sweeps, bool zero) {
        const int steps = gs_steps<DIM>(sweeps), nn = (int)L.g.nn;
        int buf = 0;
        for (int st = 0; st < steps; ++st) {
            const int col = gs_step_colour<DIM>(st), px = col & 1, py = (col >> 1) & 1, pz = (col >> 2) & 1;
            const int cx = (int)(L.g.nx - px + 1) / 2, cy = (int)(L.g.ny - py + 1) / 2;
            const int cz = DIM == 3 ? (int)(L.g.nz - pz + 1) / 2 : 1;
            int t0, mine;
            block_share(cx * cy * cz, t0, mine);
            for (int base = 0; base < mine || base == 0; base += ROUND) {
                const int cnt = max(1, min(ROUND, mine - base));
                const int combo = tid / cnt, loc = tid - combo * cnt, t = t0 + base + loc;
                const bool act = combo < W && base < mine;
                int n = 0;
                RowThird<DIM, T, false> row;
                T bv[DIM], dv[DIM], v = (T)0;
                if (act) {
                    const int q = t / cx, i = 2 * (t - q * cx) + px;
                    const int j = 2 * (DIM == 3 ? q % cy : q) + py, k = DIM == 3 ? 2 * (q / cy) + pz : 0;
                    n = i + (int)L.g.nx * (j + (int)L.g.ny * k);
                    row.load(L, n, combo / 3, combo % 3);
                    if (combo < DIM) {
#pragma unroll
                        for (int cc = 0; cc < DIM; ++cc) {
                            bv[cc] = __ldcg(L.b + cc * nn + n);
                            dv[cc] = __ldg(L.Dinv + (combo * DIM + cc) * nn + n);
                        }
                    }
                }
                T* sb = sres + buf * kCyThreads;
                if constexpr (DIM == 2) {
                    buf ^= 1;
                    bar.wait();   // (pending in the first round of the call only)
                    if (act) {
                        // the node's own value: this thread stored it in an earlier step, or another before the barrier
                        if (combo < DIM && !(zero && last_step<DIM>(st, col) < 0)) v = load_tagged(L.xt + combo * nn + n).v;
                        T part;
                        if (!row.dot_tagged(L, n, combo % 3, col, st, tag, zero, !s_dead, part)) {
                            if (!s_dead) atomicOr(a.bar + 2, 1u);
                            s_dead = 1;
                        }
                        sb[tid] = part;
                    }
                } else {
                    if (base == 0) bar.wait();
                    else __syncthreads();   // the previous round's sums have been read
                    if (act) {
                        if (combo < DIM) v = __ldcg(L.x + combo * nn + n);
                        sb[tid] = row.dot(L, n, combo % 3, L.x);
                    }
                }
                __syncthreads();
                if (act && combo < DIM) {
#pragma unroll
                    for (int cc = 0; cc < DIM; ++cc) {
                        const T* p = sb + cc * 3 * cnt + loc;
                        v = fma(dv[cc], bv[cc] - ((p[0] + p[cnt]) + p[2 * cnt]), v);
                    }
                    if (DIM == 2) store_tagged(L.xt + combo * nn + n, v, tag + 1u + (uint32_t)st);
                    L.x[combo * nn + n] = v;
                }
            }
            if (DIM == 3 || st + 1 == steps) bar.arrive();
        }
        tag += (uint32_t)steps + 2u;
    };
    auto smooth = [&](const CyLevel<T>& L, int sweeps, bool zero) {
        if (!a.cheb) {
            smooth_gs(L, sweeps, zero);
            return;
        }
        const T* cur = zero ? nullptr : L.x;
        for (int k = 0; k < sweeps; ++k) {
            T* dst = (k % 2 == 0) ? L.t : L.x;
            bar.wait();
            node_phase<DIM, T, HALF, kCheb>(L, cur, dst, L.c1[k], L.c2[k], k == 0, sres);
            bar.arrive();
            cur = dst;
        }
        if (sweeps % 2 == 1) {
            bar.wait();
            for (int i = gt; i < (int)L.g.nn * DIM; i += gn) L.x[i] = __ldcg(L.t + i);
            bar.arrive();
        }
    };

    // the cycle: down
    for (int i = gt; i < (int)a.n; i += gn) a.L[0].x[i] = (T)0;
    bar.arrive();
    for (int l = 0; l + 1 < a.nlev; ++l) {
        const CyLevel<T>&L = a.L[l], &C = a.L[l + 1];
        smooth(L, a.down, true);
        bar.wait();
        node_phase<DIM, T, HALF, kResidual>(L, L.x, L.r, (T)0, (T)0, false, sres);
        bar.sync();
        // b of the next level = P^T r (k_restrict's weights and masks), its iterate cleared
        const Grid &gf = L.g, &gc = C.g;
        for (int it = gt; it < (int)gc.nn * DIM; it += gn) {
            const int d = it / (int)gc.nn, N = it - d * (int)gc.nn;
            int64_t I, J, K;
            node_ijk<DIM>(gc, N, I, J, K);
            T acc = (T)0;
#pragma unroll
            for (int q = 0; q < nblocks<DIM>(); ++q) {
                const int dx = q % 3 - 1, dy = (q / 3) % 3 - 1, dz = DIM == 3 ? q / 9 - 1 : 0;
                const int i = 2 * (int)I + dx, j = 2 * (int)J + dy, k = 2 * (int)K + dz;
                const bool in = i >= 0 && i < gf.nx && j >= 0 && j < gf.ny && (DIM == 2 || (k >= 0 && k < gf.nz));
                const int n = (in ? i : 2 * (int)I) +
                              (int)gf.nx * ((in ? j : 2 * (int)J) + (int)gf.ny * (DIM == 3 ? (in ? k : 2 * (int)K) : 0));
                const T v = __ldcg(L.r + d * (int)gf.nn + n);
                const bool live = in && !__ldg(L.fixed + n * DIM + d);
                acc = fma((T)((dx ? 0.5 : 1.0) * (dy ? 0.5 : 1.0) * (dz ? 0.5 : 1.0)), live ? v : (T)0, acc);
            }
            C.b[it] = __ldg(C.fixed + N * DIM + d) ? (T)0 : acc;
            C.x[it] = (T)0;
        }
        bar.sync();      // the smoother may fetch b before it waits, so b is complete here
    }
    {   // coarsest level: the dense inverse, one warp per row (k_gemv)
        bar.wait();
        const CyLevel<T>& C = a.L[a.nlev - 1];
        const int lane = tid & 31, n = (int)a.ncoarse;
        for (int row = gt >> 5; row < n; row += gn >> 5) {
            double s = 0.0;
#pragma unroll 4
            for (int j = lane; j < n; j += 32) s += __ldg(a.Cinv + (int64_t)row * n + j) * (double)__ldcg(C.b + j);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) C.x[row] = (T)s;
        }
        bar.arrive();
    }
    for (int l = a.nlev - 2; l >= 0; --l) {
        // x += P x_coarse (k_prolong_add)
        const CyLevel<T>&F = a.L[l], &C = a.L[l + 1];
        const Grid &gf = F.g, &gc = C.g;
        bar.wait();
        for (int it = gt; it < (int)gf.nn * DIM; it += gn) {
            const int d = it / (int)gf.nn, n = it - d * (int)gf.nn;
            int64_t i, j, k;
            node_ijk<DIM>(gf, n, i, j, k);
            const int ox = (int)(i & 1), oy = (int)(j & 1), oz = (int)(k & 1);
            const T w = (T)((ox ? 0.5 : 1.0) * (oy ? 0.5 : 1.0) * (oz ? 0.5 : 1.0));
            T acc = (T)0;
#pragma unroll
            for (int q = 0; q < (1 << DIM); ++q) {
                const int qx = q & 1, qy = (q >> 1) & 1, qz = (q >> 2) & 1;
                const bool in = qx <= ox && qy <= oy && qz <= oz;
                const int N = (int)(i >> 1) + (in ? qx : 0) +
                              (int)gc.nx * ((int)(j >> 1) + (in ? qy : 0) + (int)gc.ny * ((int)(k >> 1) + (in ? qz : 0)));
                const T v = __ldcg(C.x + d * (int)gc.nn + N);
                const bool live = in && !__ldg(C.fixed + N * DIM + d);
                acc = fma(w, live ? v : (T)0, acc);
            }
            const T old = __ldcg(F.x + it), v = __ldg(F.fixed + n * DIM + d) ? old : old + acc;
            F.x[it] = v;
            if (DIM == 2 && !a.cheb) store_tagged(F.xt + it, v, tag);   // the smoother's initial values
        }
        bar.arrive();
        smooth(F, a.up, false);
    }
    if (!a.V) return;

    bar.wait();
    node_phase<DIM, T, false, kApply>(a.L[0], a.L[0].x, a.w, (T)0, (T)0, false, sres);
    bar.arrive();
    // Gram-Schmidt on the first kCyKrylovBlocks blocks: each keeps its chunk of w in registers of its
    // threads' strided entries (re-read from L2), every block adds up all partial sums in the same order
    const int nb = min((int)gridDim.x, kCyKrylovBlocks), m = a.k + 1, warp = tid >> 5, lane = tid & 31;
    const int chunk = ((int)a.n + nb - 1) / nb, lo = (int)blockIdx.x * chunk;
    const int len = (int)blockIdx.x < nb ? max(0, min(chunk, (int)a.n - lo)) : 0;
    auto total = [&](const double* p) {   // sum of nb partial sums by one warp
        double v = 0.0;
        for (int q = lane; q < nb; q += 32) v += __ldcg(p + q);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    for (int pass = 0; pass < 2; ++pass) {
        double* part = a.part + (int64_t)pass * kCyPass * kCyKrylovBlocks;
        bar.wait();
        if ((int)blockIdx.x < nb) {
            for (int j = warp; j < m; j += kCyThreads / 32) {
                const T* V = a.V + (int64_t)j * a.n + lo;
                LongSum<T> acc;
#pragma unroll 4
                for (int i = lane; i < len; i += 32) acc.add(V[i], __ldcg(a.w + lo + i));
                warp_merge(acc);
                if (lane == 0) part[j * kCyKrylovBlocks + blockIdx.x] = acc.value();
            }
        }
        bar.sync();
        if ((int)blockIdx.x < nb) {
            for (int j = warp; j < m; j += kCyThreads / 32) {
                const double v = total(part + j * kCyKrylovBlocks);
                if (lane == 0) s_h[j] = v;
            }
            __syncthreads();
            if (blockIdx.x == 0 && tid < m) a.out[pass * kCyPass + tid] = s_h[tid];
            LongSum<T> sq;
            for (int i = tid; i < len; i += kCyThreads) {
                const T* V = a.V + lo + i;
                T acc = __ldcg(a.w + lo + i);
#pragma unroll 4
                for (int j = 0; j < m; ++j) acc = fma((T)(-s_h[j]), V[(int64_t)j * a.n], acc);
                a.w[lo + i] = acc;
                sq.add(acc, acc);
            }
            if (pass == 1) {   // ||w||^2
                warp_merge(sq);
                __syncthreads();
                if (lane == 0) s_h[warp] = sq.value();
                __syncthreads();
                if (tid == 0) {
                    double t = 0.0;
                    for (int q = 0; q < kCyThreads / 32; ++q) t += s_h[q];
                    a.part[(int64_t)2 * kCyPass * kCyKrylovBlocks + blockIdx.x] = t;
                }
            }
        }
        bar.arrive();
    }
    bar.wait();
    if ((int)blockIdx.x < nb) {
        const double nn = total(a.part + (int64_t)2 * kCyPass * kCyKrylovBlocks);
        if (gt == 0) a.out[2 * kCyPass] = nn;
        const double hn = sqrt(nn > 0.0 ? nn : 0.0);
        if (hn > 0.0) {
            const T inv = (T)(1.0 / hn);
            for (int i = tid; i < len; i += kCyThreads) a.vnext[lo + i] = inv * __ldcg(a.w + lo + i);
        }
    }
}

template <typename T> const T* A_of(const Level& L);
template <> const double* A_of<double>(const Level& L) { return L.A64.p; }
template <> const float* A_of<float>(const Level& L) { return L.A32.p; }
template <typename T> const T* Dinv_of(const Level& L);
template <> const double* Dinv_of<double>(const Level& L) { return L.Dinv64.p; }
template <> const float* Dinv_of<float>(const Level& L) { return L.Dinv32.p; }
double* vec(DArray<double>& d, DArray<float>&, double) { return d.p; }
float* vec(DArray<double>&, DArray<float>& f, float) { return f.p; }

void prepare(Context& c) {
    if (c.cycle_bar.p) return;
    c.cycle_bar.ensure(4);
    UWG_CUDA(cudaMemsetAsync(c.cycle_bar.p, 0, 4 * sizeof(uint32_t), c.stream));
    c.cycle_part.ensure((size_t)3 * kCyPass * kCyKrylovBlocks);
}

template <int DIM, typename T, bool HALF>
void launch(Context& c, CyArgs<T>& a) {
    int sms = 0;
    UWG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
    prepare(c);
    a.bar = c.cycle_bar.p;
    a.which = c.cycle_which;
    a.part = c.cycle_part.p;
    if (DIM == 2 && !a.cheb) {
        // tagged iterates of the levels, and tags that no earlier launch has used; a word keeps the place and
        // type it had, or starts again from tag 0
        size_t bytes = 0;
        for (int l = 0; l + 1 < a.nlev; ++l) bytes += (size_t)a.L[l].g.nn * DIM * sizeof(Tagged<T>);
        const uint64_t tags = (uint64_t)a.nlev * (gs_steps<DIM>(a.down) + gs_steps<DIM>(a.up) + 4);
        const uint64_t layout[3] = {(uint64_t)a.L[0].g.nx, (uint64_t)a.L[0].g.ny, (uint64_t)a.nlev * 16 + sizeof(T)};
        const bool fresh = c.cycle_tagged.n * sizeof(uint64_t) < bytes ||
                           !std::equal(layout, layout + 3, c.cycle_layout);
        c.cycle_tagged.ensure((bytes + 15) / 16 * 2);
        if (fresh || c.cycle_tag + tags > 0xffffffffull) {
            UWG_CUDA(cudaMemsetAsync(c.cycle_tagged.p, 0, c.cycle_tagged.n * sizeof(uint64_t), c.stream));
            c.cycle_tag = 1;
            std::copy(layout, layout + 3, c.cycle_layout);
        }
        unsigned char* at = reinterpret_cast<unsigned char*>(c.cycle_tagged.p);
        for (int l = 0; l + 1 < a.nlev; ++l) {
            a.L[l].xt = reinterpret_cast<Tagged<T>*>(at);
            at += (size_t)a.L[l].g.nn * DIM * sizeof(Tagged<T>);
        }
        a.tag = (uint32_t)c.cycle_tag;
        c.cycle_tag += tags;
    }
    void* args[] = {(void*)&a};
    UWG_CUDA(cudaLaunchCooperativeKernel((const void*)k_cycle<DIM, T, HALF>, dim3((unsigned)sms), dim3(kCyThreads), args, 0,
                                         c.stream));
    c.cycle_which ^= 1;
}

template <typename T>
void fill(Context& c, const CycleOpts& o, int first, const T* b, T* x, CyArgs<T>& a) {
    a = CyArgs<T>{};
    a.nlev = c.nlevels - first;
    a.cheb = o.cheb ? 1 : 0;
    a.down = o.down;
    a.up = o.up;
    a.n = c.levels[first].mesh.nn * c.mesh.dim;
    const bool half = sizeof(T) == 4 && c.levels[0].has16 && c.smooth16;
    double bytes = 0.0, flops = 0.0;
    for (int l = first; l < c.nlevels; ++l) {
        Level& L = c.levels[l];
        CyLevel<T>& C = a.L[l - first];
        C.g = grid_of(L.mesh);
        C.A = A_of<T>(L);
        C.A16 = L.A16.p;
        C.S16 = L.S16.p;
        C.Dinv = Dinv_of<T>(L);
        C.b = l == first ? const_cast<T*>(b) : vec(L.b64, L.b32, T());
        C.x = l == first ? x : vec(L.x64, L.x32, T());
        C.r = vec(L.r64, L.r32, T());
        C.t = vec(L.t64, L.t32, T());
        C.fixed = L.fixed.p;
        // the recurrence of level_cheb
        const double lmax = 1.1 * L.lmax, lmin = 0.1 * L.lmax, theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
        const double sigma = theta / delta;
        double rho = 1.0 / sigma;
        for (int k = 0; k < kCyMaxDegree; ++k) {
            if (k == 0) {
                C.c1[0] = (T)0;
                C.c2[0] = (T)(1.0 / theta);
                continue;
            }
            const double rn = 1.0 / (2.0 * sigma - rho);
            C.c1[k] = (T)(rn * rho);
            C.c2[k] = (T)(2.0 * rn / delta);
            rho = rn;
        }
        if (l + 1 < c.nlevels) {
            const double D = L.mesh.dim, NB = D == 3 ? 27 : 9, passes = (o.cheb ? 1.0 : 2.0) * (o.down + o.up) + 1.0;
            bytes += passes * L.mesh.nn * D * D * (half ? (NB + 1) / 2 * 4 : NB * sizeof(T));
            flops += passes * 2.0 * L.mesh.nn * D * D * NB;
        }
    }
    const Level& last = c.levels[c.nlevels - 1];
    a.Cinv = last.Cinv.p;
    a.ncoarse = last.ncoarse;
    note_work(c, UWGPU_KERNEL_SMOOTH, bytes, flops);
}

template <typename T>
void run(Context& c, CyArgs<T>& a) {
    LaunchScope ls(c, UWGPU_KERNEL_SMOOTH);
    if constexpr (sizeof(T) == 4) {
        if (c.levels[0].has16 && c.smooth16) {
            if (c.mesh.dim == 3) launch<3, T, true>(c, a);
            else launch<2, T, true>(c, a);
            return;
        }
    }
    if (c.mesh.dim == 3) launch<3, T, false>(c, a);
    else launch<2, T, false>(c, a);
}

}  // namespace

int cycle_first_level(const Context& c, const CycleOpts& o) {
    const int nlev = c.nlevels;
    if (nlev < 2 || o.cycle != 1 || o.down < 0 || o.up < 0 || o.down > kCySweeps || o.up > kCySweeps) return nlev;
    if (o.cheb && (o.down > kCyMaxDegree || o.up > kCyMaxDegree || o.down < 1)) return nlev;
    if (c.levels[nlev - 1].ncoarse > 4000) return nlev;
    const int64_t limit = !o.cheb ? kCyNodesColour : c.levels[0].mesh.nn <= kCyNodesWhole ? kCyNodesWhole : kCyNodesCheb;
    int first = nlev - 1;
    while (first > 0 && nlev - first < kCyMaxLevels && c.levels[first - 1].mesh.nn <= limit) --first;
    return first == nlev - 1 ? nlev : first;
}

template <typename T>
void cycle_run(Context& c, const CycleOpts& o, int first, const T* b, T* x) {
    CyArgs<T> a;
    fill<T>(c, o, first, b, x, a);
    run<T>(c, a);
}

template <typename T>
void cycle_fgmres_iteration(Context& c, const CycleOpts& o, const T* V, int k, int64_t n, T* z, T* w, T* vnext,
                            double* host_out) {
    CyArgs<T> a;
    fill<T>(c, o, 0, V + (int64_t)k * n, z, a);
    a.V = V;
    a.vnext = vnext;
    a.w = w;
    a.k = k;
    a.out = host_out;
    run<T>(c, a);
}

void cycle_begin(Context& c) {
    if (c.cycle_give_up) prepare(c);
    if (c.cycle_bar.p)
        UWG_CUDA(cudaMemsetAsync(c.cycle_bar.p + 2, c.cycle_give_up ? 1 : 0, sizeof(uint32_t), c.stream));
    c.cycle_give_up = false;
}

void cycle_check(Context& c) {
    if (!c.cycle_bar.p) return;
    uint32_t err = 0;
    UWG_CUDA(cudaMemcpyAsync(&err, c.cycle_bar.p + 2, sizeof(err), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    if (err) {
        UWG_CUDA(cudaMemsetAsync(c.cycle_bar.p, 0, 4 * sizeof(uint32_t), c.stream));
        throw Error(UWGPU_ERR_CUDA, "multigrid cycle: a grid barrier did not complete in time");
    }
}

template void cycle_run<double>(Context&, const CycleOpts&, int, const double*, double*);
template void cycle_run<float>(Context&, const CycleOpts&, int, const float*, float*);
template void cycle_fgmres_iteration<double>(Context&, const CycleOpts&, const double*, int, int64_t, double*, double*,
                                             double*, double*);
template void cycle_fgmres_iteration<float>(Context&, const CycleOpts&, const float*, int, int64_t, float*, float*, float*,
                                            double*);

}  // namespace uwg
