// Jacobi-preconditioned CG on G^T W G (3D, FP32, matrix-free from the folded nodal weights; see
// gwg_stencil.cu) as one cooperative launch for the whole solve.
//
// Launched as two kernels per iteration (direction and update), the CG is bound by the launches and by
// re-reading its vectors from L2: on a 64 x 80 x 112 mesh an iteration moves 27 MB and takes 12 us.  Here
// the mesh is cut into bricks, one per block and at most one block per SM, and a brick's vectors never
// leave the block: r, p and q of up to eight elements (a piece of a z column) and the weights of their
// nodes are in a thread's registers, x and 1/diag of its elements, z with its halo and the weighted gradients
// at the nodes in shared memory.  Per iteration the blocks exchange only
//   - z of the elements on brick faces, as 64-bit words {value, tag}: a reader polls the word until the
//     tag is the iteration's, so the exchange needs no barrier of its own and no fence;
//   - the block sums of r.z and p.q, as words of the same kind that every block reads and adds in the same
//     order.  Each is also the barrier that makes the words of the iteration before free to be overwritten:
//     a block publishes its p.q only after it has read its halo and every r.z, and its r.z only after every
//     p.q.
// The sums are exchanged by a warp of their own.  beta does not enter A z, so the other warps read the halo and
// form A z while that warp waits for r.z; they wait for p.q.  An iteration is then bound by that one wait (a
// store, its way through L2, the load that sees it and the sums: 1 to 2 us, growing with the blocks that poll),
// the halo's, and the shared-memory reads of the stencil.  Measured per iteration, with the sums in pairs of FP32
// (below), two launches -> one warp of sixteen exchanging while the others wait -> this form: 64 x 80 x 112
// elements 12.3 -> 7.5 -> 7.1 us, 64^3 8.3 -> 6.0 -> 5.1, 32^3 -> 4.9 -> 3.6, 16^3 -> 3.7 -> 3.2.  Sixteen copies
// of the block sums, so that the blocks do not all poll the same lines: 8.2 -> 7.5 us on the first mesh.
//
// A thread's and a warp's sums are FP32 and all sums above a warp FP64, as in the two-kernel form: a sum over the
// mesh may pass the largest FP32.  The thirteen dependent FP64 additions of a sum hold its warp for 64 cycles each;
// as pairs of FP32 (48 bits, FP32 range) the same sums took 0.7 to 1.0 us less per iteration.  That is the price of
// the precision: per iteration now 64 x 80 x 112 elements 7.9 us, 64^3 5.8, 32^3 4.6, 16^3 4.0.  (Additions with
// half the lanes off at each level, and a division by an FP32 reciprocal and two corrections, gain nothing.)
//
// Every wait is bounded; a block whose wait ends without its word reports an error and returns.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "internal.cuh"

namespace uwg {

namespace {

constexpr int kWt = 512;                 // threads that hold elements and nodes
constexpr int kWWarps = kWt / 32;        // the warp after them exchanges the sums
constexpr int kWAll = kWt + 32;
constexpr int kWSeg = 8;                 // elements per thread at most
constexpr int kWRim = 3;                 // nodes of the brick's upper faces per thread at most
constexpr int kWHalo = 4;                // halo elements per thread at most
constexpr int kWBlocks = 160;            // blocks at most: five sums per lane
constexpr int kWCopies = 16;             // copies of the block sums, each read by a sixteenth of the blocks
static_assert(kWCopies <= 32 && kWWarps == 16, "one lane per word published, each holding the block's sum");
constexpr int kWCheck = 12;              // iterations between convergence tests, as in the two-kernel form
constexpr int kWPoll = 1 << 20;

typedef uint64_t u64;

struct CgWhole {
    int ex, ey, ez;
    int bx, by, bz;                      // largest brick
    int nbx, nby, nbz;
    int seg;                             // elements per thread
    int hx, hxy, nflat;                  // row and plane of z with halo; nodes, numbered with the same pitches
    int halo;                            // halo elements of the largest brick
    int64_t pitch, nny, nn;              // weights [d][node plane][y][pitch], entries per d
    const float* Wc;
    const float* dinv;
    const double* b;
    float* x;
    u64* face;                           // [element] {z, tag}
    u64* sums;                           // [rz, pq, rr][copy][block] {sum, tag}
    double* report;                      // iterations, code, ||r||, ||b||
    int* failed;
    int maxit;
    double rtol;
};

__device__ __forceinline__ void st_word(u64* p, float v, uint32_t tag) {
    const u64 w = ((u64)tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ u64 ld_word(const u64* p) {
    u64 w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}
// a block sum and its tag in one aligned 16-byte word, read and written whole
__device__ __forceinline__ void st_sum(u64* p, double v, uint32_t tag) {
    asm volatile("{ .reg .b128 q; mov.b128 q, {%1, %2}; st.relaxed.gpu.global.b128 [%0], q; }" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((u64)tag)
                 : "memory");
}
__device__ __forceinline__ void ld_sum(const u64* p, double& v, uint32_t& tag) {
    u64 a, b;
    asm volatile("{ .reg .b128 q; ld.relaxed.gpu.global.b128 q, [%2]; mov.b128 {%0, %1}, q; }" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    v = __longlong_as_double((long long)a);
    tag = (uint32_t)b;
}
__device__ __forceinline__ float word_value(u64 w) { return __uint_as_float((uint32_t)w); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// exchange warp: publishes the sum of the block's warp sums sw and adds those of all blocks, every lane of every
// block in the same order; false when a word does not come
__device__ __forceinline__ bool global_sum(const float* sw, u64* slots, int blocks, uint32_t tag, double& sum) {
    const int lane = threadIdx.x & 31;
    double v = (double)sw[lane % kWWarps];   // the two halves of the warp form the same sum
#pragma unroll
    for (int o = kWWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane < kWCopies) st_sum(slots + 2 * (kWBlocks * lane + blockIdx.x), v, tag);
    const u64* from = slots + 2 * kWBlocks * (blockIdx.x % kWCopies);
    constexpr int M = kWBlocks / 32;
    double w[M];
    uint32_t t[M];
    bool all = false;
    for (int tries = 0; tries < kWPoll && !all; ++tries) {
        bool mine = true;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int i = lane + 32 * m;
            w[m] = 0.0;
            t[m] = tag;
            if (i < blocks) ld_sum(from + 2 * i, w[m], t[m]);
        }
#pragma unroll
        for (int m = 0; m < M; ++m) mine = mine && t[m] == tag;
        all = __all_sync(0xffffffffu, mine);
    }
    v = w[0];
#pragma unroll
    for (int m = 1; m < M; ++m) v += w[m];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    sum = v;
    return all;
}

// barrier of the whole block, and of the warps that hold elements
__device__ __forceinline__ void sync_all() { asm volatile("bar.sync 0, %0;" ::"n"(kWAll) : "memory"); }
__device__ __forceinline__ void sync_work() { asm volatile("bar.sync 1, %0;" ::"n"(kWt) : "memory"); }

template <int SEG>
__global__ void __launch_bounds__(kWAll, 1) k_cg_whole(CgWhole a) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float sw[kWWarps], sw2[kWWarps];
    __shared__ float s_alpha, s_beta;
    __shared__ int s_stop, s_fail, s_halo;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int zsize = a.nflat + (SEG + 1) * a.hxy + a.hx + 2;   // and what short pieces of the last plane read
    float* zb = smem;                                        // z, elements of the brick from (1, 1, 1)
    float* yb = zb + zsize;                                  // [3][node]
    const int ysize = 3 * a.nflat + SEG * a.hxy + a.hx + 2;  // likewise
    float* xs = yb + ysize;                                  // x, [element of the thread][thread]
    float* ds = xs + SEG * kWt;                              // 1/diag, the same
    uint2* list = reinterpret_cast<uint2*>(ds + SEG * kWt + ((zsize + ysize) & 1));   // {place in zb, element}
    const int ix = blockIdx.x % a.nbx, iy = blockIdx.x / a.nbx % a.nby, iz = blockIdx.x / (a.nbx * a.nby);
    const int x0 = ix * a.bx, y0 = iy * a.by, z0 = iz * a.bz;
    const int cx = min(a.bx, a.ex - x0), cy = min(a.by, a.ey - y0), cz = min(a.bz, a.ez - z0);   // this brick
    if (tid == 0) {
        s_stop = 0;
        s_fail = 0;
        s_halo = 0;
    }
    for (int i = tid; i < zsize; i += kWAll) zb[i] = 0.f;
    __syncthreads();
    // halo elements inside the mesh (the others stay zero)
    for (int i = tid; i < (cz + 2) * (cy + 2) * (cx + 2); i += kWAll) {
        const int hx = i % (cx + 2), t = i / (cx + 2), hy = t % (cy + 2), hz = t / (cy + 2);
        const bool inner = hx >= 1 && hx <= cx && hy >= 1 && hy <= cy && hz >= 1 && hz <= cz;
        const int gx = x0 + hx - 1, gy = y0 + hy - 1, gz = z0 + hz - 1;
        if (!inner && gx >= 0 && gx < a.ex && gy >= 0 && gy < a.ey && gz >= 0 && gz < a.ez)
            list[atomicAdd(&s_halo, 1)] = make_uint2((unsigned)(hx + a.hx * hy + a.hxy * hz),
                                                     (unsigned)(gx + a.ex * (gy + a.ey * gz)));
    }
    u64* rz_slots = a.sums;
    u64* pq_slots = rz_slots + 2 * kWBlocks * kWCopies;
    u64* rr_slots = pq_slots + 2 * kWBlocks * kWCopies;
    const int blocks = gridDim.x;
    // k = -1: z = 1/diag b, p = z, q = A z; then iteration k: x, r, z with alpha, r.z, p and q with beta, p.q
    if (warp == kWWarps) {
        double rz = 0.0, norm0 = 0.0;
        sync_all();
        for (int k = -1;; ++k) {
            const uint32_t tag = (uint32_t)(k + 2);
            const bool check = k < 0 || (k + 1) % kWCheck == 0;
            sync_all();
            double rz_new, pq, rr = 0.0;
            bool ok = global_sum(sw, rz_slots, blocks, tag, rz_new);
            if (check) ok = global_sum(sw2, rr_slots, blocks, tag, rr) && ok;
            if (lane == 0) {
                s_beta = k < 0 ? 0.f : (float)(rz_new / rz);
                if (!ok) s_fail = 1;
                if (check) {
                    const double norm = sqrt(rr);
                    if (k < 0) norm0 = norm;
                    const int code = !(norm0 > 0.0) ? 1 : !isfinite(norm) ? 2 : k >= 0 && norm <= a.rtol * norm0 ? 3
                                   : k + 1 >= a.maxit ? 4 : 0;
                    s_stop = code;
                    if (code && blockIdx.x == 0) {
                        a.report[0] = k + 1;
                        a.report[1] = code;
                        a.report[2] = norm;
                        a.report[3] = norm0;
                    }
                }
            }
            rz = rz_new;
            sync_all();
            if (s_fail || s_stop) break;
            sync_all();
            ok = global_sum(sw, pq_slots, blocks, tag, pq);
            if (lane == 0) {
                s_alpha = (float)(rz / pq);
                if (!ok) s_fail = 1;
            }
            sync_all();
            if (s_fail) break;
        }
        if (s_fail && lane == 0) atomicExch(a.failed, 1);
        return;
    }
    // this thread's elements: `cnt` of the column (tx, ty) from plane tz
    const int cols = a.bx * a.by, col = tid % cols, tx = col % a.bx, ty = col / a.bx, tz = tid / cols * a.seg;
    const int cnt = tx < cx && ty < cy ? max(0, min(a.seg, cz - tz)) : 0;
    const int e0 = (x0 + tx) + a.ex * ((y0 + ty) + a.ey * (z0 + tz)), exy = a.ex * a.ey;
    const int n0 = cnt > 0 ? tx + a.hx * ty + a.hxy * tz : 0;   // lower corner node of the first
    const int c0 = n0 + 1 + a.hx + a.hxy;
    float r[SEG], p[SEG], q[SEG];
    unsigned faces = 0;
#pragma unroll
    for (int j = 0; j < SEG; ++j) {
        const bool in = j < cnt;
        r[j] = in ? (float)a.b[e0 + j * exy] : 0.f;
        ds[j * kWt + tid] = in ? a.dinv[e0 + j * exy] : 0.f;
        p[j] = q[j] = 0.f;
        xs[j * kWt + tid] = 0.f;
        if (in && (tx == 0 || tx == cx - 1 || ty == 0 || ty == cy - 1 || tz + j == 0 || tz + j == cz - 1)) faces |= 1u << j;
    }
    // weights of its nodes: the lower corner node of each of its elements, and some nodes on the upper faces
    // of the brick (x = cx, then y = cy, then z = cz)
    auto weight = [&](int nx, int ny, int nz, bool in, float* to) {
        const int64_t o = in ? (x0 + nx) + a.pitch * ((y0 + ny) + a.nny * (int64_t)(z0 + nz)) : 0;
        for (int k = 0; k < 3; ++k) to[k] = in ? __ldg(a.Wc + k * a.nn + o) : 0.f;
    };
    float w[SEG][3], wr[kWRim][3];
    int rim[kWRim];
#pragma unroll
    for (int j = 0; j < SEG; ++j) weight(tx, ty, tz + j, j < cnt, w[j]);
    const int fx = (cy + 1) * (cz + 1), fy = cx * (cz + 1), fz = cx * cy;
#pragma unroll
    for (int m = 0; m < kWRim; ++m) {
        int i = tid + m * kWt, nx, ny, nz;
        const bool in = i < fx + fy + fz;
        if (i < fx) {
            nx = cx;
            ny = i % (cy + 1);
            nz = i / (cy + 1);
        } else if ((i -= fx) < fy) {
            nx = i % cx;
            ny = cy;
            nz = i / cx;
        } else {
            i -= fy;
            nx = i % cx;
            ny = i / cx;
            nz = cz;
        }
        rim[m] = in ? nx + a.hx * ny + a.hxy * nz : -1;
        weight(nx, ny, nz, in, wr[m]);
    }
    sync_all();
    const int nh = s_halo;
    for (int k = -1;; ++k) {
        const uint32_t tag = (uint32_t)(k + 2);
        {
            const float alpha = k < 0 ? 0.f : s_alpha;
            float rz = 0.f, rr = 0.f;
#pragma unroll
            for (int j = 0; j < SEG; ++j)
                if (j < cnt) {
                    if (k >= 0) {
                        xs[j * kWt + tid] = fmaf(alpha, p[j], xs[j * kWt + tid]);
                        r[j] = fmaf(-alpha, q[j], r[j]);
                    }
                    const float z = r[j] * ds[j * kWt + tid];
                    zb[c0 + j * a.hxy] = z;
                    if (faces >> j & 1u) st_word(a.face + e0 + j * exy, z, tag);
                    rz = fmaf(r[j], z, rz);
                    rr = fmaf(r[j], r[j], rr);
                }
            rz = warp_sum(rz);
            if (k < 0 || (k + 1) % kWCheck == 0) rr = warp_sum(rr);
            if (lane == 0) {
                sw[warp] = rz;
                sw2[warp] = rr;
            }
        }
        sync_all();
        // while the exchange warp waits for r.z: the halo, and A z, which beta does not enter
        {
            u64 v[kWHalo];
            uint2 at[kWHalo];
#pragma unroll
            for (int m = 0; m < kWHalo; ++m) at[m] = tid + m * kWt < nh ? list[tid + m * kWt] : make_uint2(0xffffffffu, 0u);
            bool all = false;
            for (int tries = 0; tries < kWPoll && !all; ++tries) {
                all = true;
#pragma unroll
                for (int m = 0; m < kWHalo; ++m)
                    if (at[m].x != 0xffffffffu) v[m] = ld_word(a.face + at[m].y);
#pragma unroll
                for (int m = 0; m < kWHalo; ++m)
                    if (at[m].x != 0xffffffffu) all = all && (uint32_t)(v[m] >> 32) == tag;
            }
#pragma unroll
            for (int m = 0; m < kWHalo; ++m)
                if (at[m].x != 0xffffffffu) zb[at[m].x] = word_value(v[m]);
            if (!all) s_fail = 1;
        }
        sync_work();
        // nodes: y_d = W_d (sum of z above the node along d - sum below).  A thread's own nodes lie above one
        // another and share the sums of an element plane: 4 + 3 shared-memory accesses each instead of 8 + 3
        {
            float gx = 0.f, gy = 0.f, z00 = 0.f, z10 = 0.f, z01 = 0.f, z11 = 0.f;
#pragma unroll
            for (int j = 0; j <= SEG; ++j) {   // of a short piece the planes above it are read and not used
                const float* f = zb + n0 + j * a.hxy;
                const float f00 = f[0], f10 = f[1], f01 = f[a.hx], f11 = f[a.hx + 1];
                const float hx = (f10 - f00) + (f11 - f01), hy = (f01 - f00) + (f11 - f10);
                if (j > 0 && j <= cnt) {
                    float* y = yb + n0 + (j - 1) * a.hxy;
                    y[0] = w[j - 1][0] * (gx + hx);
                    y[a.nflat] = w[j - 1][1] * (gy + hy);
                    y[2 * a.nflat] = w[j - 1][2] * (((f00 - z00) + (f10 - z10)) + ((f01 - z01) + (f11 - z11)));
                }
                gx = hx;
                gy = hy;
                z00 = f00;
                z10 = f10;
                z01 = f01;
                z11 = f11;
            }
        }
#pragma unroll
        for (int m = 0; m < kWRim; ++m)
            if (rim[m] >= 0) {
                const float* f = zb + rim[m];
                const float* g = f + a.hxy;
                float* y = yb + rim[m];
                const float z000 = f[0], z100 = f[1], z010 = f[a.hx], z110 = f[a.hx + 1];
                const float z001 = g[0], z101 = g[1], z011 = g[a.hx], z111 = g[a.hx + 1];
                y[0] = wr[m][0] * (((z100 - z000) + (z110 - z010)) + ((z101 - z001) + (z111 - z011)));
                y[a.nflat] = wr[m][1] * (((z010 - z000) + (z110 - z100)) + ((z011 - z001) + (z111 - z101)));
                y[2 * a.nflat] = wr[m][2] * (((z001 - z000) + (z101 - z100)) + ((z011 - z010) + (z111 - z110)));
            }
        sync_work();
        // elements: A z from the two node planes of each, the lower one kept from the element below
        float az[SEG];
        {
            float lo_xy = 0.f, lo_z = 0.f;
#pragma unroll
            for (int j = 0; j <= SEG; ++j) {   // planes above a short piece are read and not used
                const float* y = yb + n0 + j * a.hxy;
                const float* y1 = y + a.nflat;
                const float* y2 = y1 + a.nflat;
                const float gx = (y[0] - y[1]) + (y[a.hx] - y[a.hx + 1]);
                const float gy = (y1[0] - y1[a.hx]) + (y1[1] - y1[a.hx + 1]);
                const float gz = (y2[0] + y2[1]) + (y2[a.hx] + y2[a.hx + 1]);
                if (j > 0) az[j - 1] = (lo_xy + (gx + gy)) + (lo_z - gz);
                lo_xy = gx + gy;
                lo_z = gz;
            }
        }
        sync_all();
        if (s_fail || s_stop) break;
        const float beta = s_beta;
        float pq = 0.f;
#pragma unroll
        for (int j = 0; j < SEG; ++j)
            if (j < cnt) {
                p[j] = fmaf(beta, p[j], zb[c0 + j * a.hxy]);
                q[j] = fmaf(beta, q[j], az[j]);
                pq = fmaf(p[j], q[j], pq);
            }
        pq = warp_sum(pq);
        if (lane == 0) sw[warp] = pq;
        sync_all();
        sync_all();
        if (s_fail) break;
    }
    if (s_fail) return;
#pragma unroll
    for (int j = 0; j < SEG; ++j)
        if (j < cnt) a.x[e0 + j * exy] = xs[j * kWt + tid];
}

// the instance of the kernel: elements per thread, rounded up to a power of two
int seg_of(const CgWhole& a) { return a.seg <= 1 ? 1 : a.seg <= 2 ? 2 : a.seg <= 4 ? 4 : kWSeg; }
const void* kernel_of(const CgWhole& a) {
    switch (seg_of(a)) {
        case 1: return (const void*)k_cg_whole<1>;
        case 2: return (const void*)k_cg_whole<2>;
        case 4: return (const void*)k_cg_whole<4>;
        default: return (const void*)k_cg_whole<kWSeg>;
    }
}

// Cuts the mesh into bricks for `sms` blocks at most.  Among the cuts whose brick fits a block (elements,
// nodes and halo per thread as above) the one with the least work per thread, weighed by instructions:
// 40 per node of the upper faces, 70 per element with its lower corner node, 30 per halo element.  False when no cut fits.
bool cut(CgWhole& a, int sms, size_t* smem) {
    double best = 1e300;
    if (sms > kWBlocks) sms = kWBlocks;
    for (int nx = 1; nx <= a.ex && nx <= sms; ++nx) {
        const int bx = (a.ex + nx - 1) / nx, mx = (a.ex + bx - 1) / bx;
        if (mx != nx) continue;
        for (int ny = 1; ny <= a.ey && nx * ny <= sms; ++ny) {
            const int by = (a.ey + ny - 1) / ny, my = (a.ey + by - 1) / by;
            if (my != ny || bx * by > kWt) continue;
            for (int nz = 1; nz <= a.ez && nx * ny * nz <= sms; ++nz) {
                const int bz = (a.ez + nz - 1) / nz, mz = (a.ez + bz - 1) / bz;
                if (mz != nz) continue;
                const int pieces = kWt / (bx * by), seg = (bz + pieces - 1) / pieces;
                const int nflat = (bz + 1) * (by + 2) * (bx + 2);
                const int halo = (bx + 2) * (by + 2) * (bz + 2) - bx * by * bz;
                const int rim = (bx + 1) * (by + 1) * (bz + 1) - bx * by * bz;
                if (seg > kWSeg || rim > kWRim * kWt || halo > kWHalo * kWt) continue;
                const double cost = 40.0 * ((rim + kWt - 1) / kWt) + 70.0 * (seg + 1) * (bx % 32 ? 1.2 : 1.0) +
                                    30.0 * ((halo + kWt - 1) / kWt) + 0.01 * nx * ny * nz;
                if (cost < best) {
                    best = cost;
                    a.bx = bx;
                    a.by = by;
                    a.bz = bz;
                    a.nbx = nx;
                    a.nby = ny;
                    a.nbz = nz;
                    a.seg = seg;
                    a.hx = bx + 2;
                    a.hxy = (bx + 2) * (by + 2);
                    a.nflat = nflat;
                    a.halo = halo;
                }
            }
        }
    }
    if (best == 1e300) return false;
    const size_t n = seg_of(a);
    *smem = sizeof(float) * (4 * (size_t)a.nflat + (2 * n + 1) * a.hxy + 2 * (size_t)a.hx + 5 + 2 * n * kWt) +
            sizeof(uint2) * a.halo;
    return true;
}

}  // namespace

namespace {
bool plan(Context& c, CgWhole& a, size_t* smem) {
    const MeshDesc& m = c.levels[0].mesh;
    if (m.dim != 3 || m.ne >= ((int64_t)1 << 31)) return false;
    int sms = 0, coop = 0, optin = 0;
    UWG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
    UWG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device));
    UWG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    if (!coop) return false;
    a.ex = (int)m.nel[0];
    a.ey = (int)m.nel[1];
    a.ez = (int)m.nel[2];
    return cut(a, sms, smem) && *smem + 1024 <= (size_t)optin;
}
}  // namespace

// whether gwg_cg_whole solves on the context's mesh
bool gwg_cg_whole_fits(Context& c) {
    CgWhole a{};
    size_t smem = 0;
    return plan(c, a, &smem);
}

// Solves G^T W G x = b as gwg_cg32_mf describes.  Returns the iterations taken, or -1 when the mesh has no
// cut into bricks that fit (more than about 600,000 elements on 152 SMs).
int gwg_cg_whole(Context& c, const float* Wc, const float* dinv, const double* b, float* x, double rtol, int maxit) {
    const MeshDesc& m = c.levels[0].mesh;
    CgWhole a{};
    size_t smem = 0;
    if (!plan(c, a, &smem)) return -1;
    a.pitch = (m.nnx + 3) / 4 * 4;
    a.nny = m.nny;
    a.nn = a.pitch * m.nny * m.nnz;
    a.Wc = Wc;
    a.dinv = dinv;
    a.b = b;
    a.x = x;
    a.maxit = maxit;
    a.rtol = rtol;
    // words of the exchange: zeroed, so that no tag (from 1) of an earlier solve is left
    const size_t face = ((size_t)m.ne + 15) / 16 * 16, words = face + 6 * kWBlocks * kWCopies + 8;
    c.cg_words.ensure(words);
    UWG_CUDA(cudaMemsetAsync(c.cg_words.p, 0, words * sizeof(u64), c.stream));
    a.face = c.cg_words.p;
    a.sums = c.cg_words.p + face;   // on 128 bytes
    a.report = reinterpret_cast<double*>(a.sums + 6 * kWBlocks * kWCopies);
    a.failed = reinterpret_cast<int*>(a.report + 4);
    UWG_CUDA(cudaFuncSetAttribute(kernel_of(a), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    {
        LaunchScope ls(c, UWGPU_KERNEL_SCHUR_PC);
        void* args[] = {(void*)&a};
        UWG_CUDA(cudaLaunchCooperativeKernel(kernel_of(a), dim3((unsigned)(a.nbx * a.nby * a.nbz)), dim3(kWAll),
                                             args, smem, c.stream));
    }
    double* h = c.host_scalars;
    UWG_CUDA(cudaMemcpyAsync(h, a.report, 5 * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    int failed = 0;
    std::memcpy(&failed, h + 4, sizeof(int));
    if (failed || h[1] == 0.0) throw Error(UWGPU_ERR_CUDA, "BFBt inner solve: an exchange between blocks did not complete");
    if (h[1] == 2.0) throw Error(UWGPU_ERR_NAN, "NaN in the BFBt inner solve");
    const int it = (int)h[0];
    // traffic as of the two-kernel form's vectors; they stay on chip here
    note_work(c, UWGPU_KERNEL_SCHUR_PC, (double)m.ne * (8 + 4 + 4) + (double)m.nn * 12, (double)it * m.ne * 110.0);
    return it;
}

}  // namespace uwg
