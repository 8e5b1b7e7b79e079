// Learned velocity preconditioner: a 3D U-Net on the nodal grid (BF16 weights and activations,
// FP32 accumulation and gradients), with its own forward, backward and Adam kernels.
//
// Input channels per node: the three components of the residual r and of the multigrid
// V-cycle's answer V(r) (each scaled to unit RMS), and log10 of the node-averaged viscosity;
// output: the correction to add to V(r), in units of RMS(V(r)).  The node
// grid (nel+1 per axis) is zero-padded to a multiple of 2^(levels-1).  Level l has base * 2^l
// channels; each level is two 3x3x3 convolutions with ReLU, levels are joined by 2x2x2 average
// pooling on the way down and nearest upsampling + concatenation with the skip on the way up, and
// a 1x1x1 convolution maps the finest decoder output to the three velocity components.
//
// Layout: channels-last (voxel-major, channel fastest) so that one 16-byte load brings eight BF16
// channels of a voxel.  Weights of a 3x3x3 layer are W[tap][cin][cout]; the data-gradient pass
// runs the forward kernel on W'[tap][cout][cin] = W[26 - tap][cin][cout].
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.cuh"
#include "tc.cuh"
#include "unet.cuh"

namespace uwg {
namespace unet {

typedef __nv_bfloat16 bf16;

// ------------------------------------------------------------------------------------------
// Kernels
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void load8(const bf16* p, float v[8]) {
    uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float2 f = __bfloat1622float2(h[k]);
        v[2 * k] = f.x;
        v[2 * k + 1] = f.y;
    }
}
__device__ __forceinline__ void load8(const float* p, float v[8]) {
    float4 a = *reinterpret_cast<const float4*>(p);
    float4 b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(bf16* p, const float v[8]) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}
__device__ __forceinline__ void store8(float* p, const float v[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// ---- tensor-core (tcgen05) forms of the 3x3x3 convolution --------------------------------------
// FP32 values enter a BF16 product as two parts, hi = bf16(x) and lo = bf16(x - hi), whose sum
// carries about 16 significant bits (the split of Henry, Tang and Heinecke, "Leveraging the
// bfloat16 artificial intelligence datatype for higher-precision computations", ARITH 2019);
// both parts are multiplied on the tensor core and accumulated in FP32.
__device__ __forceinline__ void split8(const float v[8], uint4& hi, uint4& lo) {
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&hi);
    __nv_bfloat162* l = reinterpret_cast<__nv_bfloat162*>(&lo);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
        const float2 af = __bfloat1622float2(a);
        h[k] = a;
        l[k] = __floats2bfloat162_rn(v[2 * k] - af.x, v[2 * k + 1] - af.y);
    }
}

// Both convolution kernels work on tiles of 8 voxels in x by some rows in y of one z plane and
// stage, per chunk of 8 channels, the tile with its halo as [y][x] rows of 16 bytes.  Eight
// consecutive x of a row are then one 128-byte core matrix and consecutive y are a fixed stride
// apart, so the operand of a tap (dx, dy) is the staged tile at a shifted start address: a tile is
// read 4.2 times (three z planes of 10 x 18 for 8 x 16) instead of once per tap.  Staging is by
// 16-byte cp.async with zero fill outside the grid, into a ring of stages.
constexpr int kTx = 8, kTy = 16, kHx = kTx + 2;
constexpr int kConvThreads = 256;
constexpr int kConvStages = 4;                   // most stages of a ring
constexpr size_t kSmemTwo = 108 * 1024;          // dynamic shared memory with which two CTAs share an SM
constexpr size_t kSmemOne = 216 * 1024;
constexpr size_t kSmemWidth = 227 * 1024 - 64;    // see conv_launch_tc

// rows of a chunk, padded so that the 16-byte stores of eight consecutive threads (channels
// fastest, `kc8` chunks) fall in different banks
__host__ __device__ inline int chunk_rows(int rows, int kc8) {
    const int w = kc8 >= 8 ? 1 : 8 / kc8;
    return rows + ((w - rows) % 8 + 8) % 8;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// at most `ahead` (0, 1 or 2) of this thread's groups still in flight
__device__ __forceinline__ void cp_wait(int ahead) {
    if (ahead == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
    else if (ahead == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 2;" ::: "memory");
}
// stages of a ring that loads `ahead` stages before the one being multiplied: with one more stage
// than that, the load waits for the MMAs just issued; with two more, for those before
__host__ __device__ inline int ring_ahead(int stages) { return stages >= 4 ? 2 : stages >= 2 ? 1 : 0; }

// completion of the stages of a ring, in order; every wait is bounded
struct RingWait {
    uint64_t* bar;
    int stages;
    int done = 0, slot = 0;   // stages known complete, slot of the next
    uint32_t parity = 0;
    __device__ __forceinline__ bool upto(int i, uint32_t limit = 1u << 22) {
        bool ok = true;
        for (; done <= i; ++done) {
            ok = tc::mbar_wait(&bar[slot], parity, limit) && ok;
            if (++slot == stages) {
                slot = 0;
                parity ^= 1u;
            }
        }
        return ok;
    }
};

// Plan of k_conv3_tc.  A stage is the input of nine taps (one z plane of the halo) or three (one
// y shift of it, where nine do not fit) and, unless the weights of all taps stay resident, these
// taps' weights.
struct ConvPlan {
    int kc8;             // chunks of 8 input channels (even: K is padded to 16)
    int Nc, nchunks;     // output channels per CTA, and CTAs (grid.y) that share the channels
    int taps;            // 9 or 3
    int stages, resident;
    uint32_t chunkA, chunkB, partA, tapB, stage;   // bytes
    size_t smem;
};
inline bool conv_plan_try(ConvPlan& p, int K, int parts, int taps, bool resident, int least, int most, size_t budget) {
    p.kc8 = (K + 15) / 16 * 2;
    p.taps = taps;
    p.resident = resident;
    p.chunkA = (uint32_t)chunk_rows((taps == 9 ? kTy + 2 : kTy) * kHx, p.kc8) * 16u;
    p.chunkB = (uint32_t)chunk_rows(p.Nc, p.kc8) * 16u;
    p.partA = p.kc8 * p.chunkA;
    p.tapB = p.kc8 * p.chunkB;
    p.stage = (uint32_t)parts * p.partA + (resident ? 0u : (uint32_t)taps * p.tapB);
    const size_t fixed = resident ? (size_t)27 * p.tapB : 0;
    if (fixed >= budget) return false;
    const int64_t n = (int64_t)((budget - fixed) / p.stage);
    p.stages = (int)(n < most ? n : most);
    p.smem = fixed + (size_t)p.stages * p.stage;
    return p.stages >= least;
}
// `tiles` voxel tiles on `sms` SMs.  The output channels are shared out (16 at least per CTA)
// while there are fewer than two CTAs per SM: the coarse levels have 7 or 28 tiles (128 -> 128 channels on
// 7 x 7 x 7 voxels: 153 us on three CTAs, 16 us on 56).  Weights stay resident where a CTA runs over several
// tiles.  Nine taps per stage read the halo once; three where two stages of nine do not fit.
inline ConvPlan conv_plan(int K, int N, int parts, int64_t tiles, int sms) {
    const int n16 = (N + 15) / 16;
    int want = (int)((2 * (int64_t)sms + tiles - 1) / tiles);
    if (want > n16) want = n16;
    ConvPlan p;
    for (int pass = 0; pass < 2; ++pass)   // two stages at least, by narrower chunks if need be; else one
        for (int nch = want; nch <= n16; ++nch) {
            p.Nc = (n16 + nch - 1) / nch * 16;
            p.nchunks = (N + p.Nc - 1) / p.Nc;
            if (pass == 0) {
                const bool many = tiles * p.nchunks > sms;
                if (many && conv_plan_try(p, K, parts, 9, true, 3, kConvStages, kSmemTwo)) return p;
                if (many && conv_plan_try(p, K, parts, 9, true, 2, kConvStages, kSmemOne)) return p;
                if (conv_plan_try(p, K, parts, 9, false, 2, kConvStages, kSmemOne)) return p;
                if (conv_plan_try(p, K, parts, 3, false, 2, kConvStages, kSmemOne)) return p;
            } else if (conv_plan_try(p, K, parts, 3, false, 1, 1, kSmemOne)) {
                return p;
            }
        }
    throw Error(UWGPU_ERR_ARGUMENT, "tensor-core kernel: shared memory plan too large");
}

// 3x3x3 convolution as an implicit GEMM on the tensor core: for a tile of 8 x 16 voxels (rows,
// M = 128) and Nc output channels, D = sum over the 27 taps t of A_t B_t^T, with
// A_t[m][k] = in[v_m + off(t)][k] (zero outside the grid) and B_t[n][k] = W_t[k][n], read from the
// layer's other packing Wrev[26 - t][n][k] (for the forward pass the flipped transpose, for the
// data gradient the plain weights).  Operands are K-major in shared memory; the accumulator
// (128 x Nc FP32) lives in TMEM; one thread issues the MMAs of a stage while the next ones are
// loaded.  The epilogue adds the bias, applies ReLU and stores BF16 (or FP32) rows.  CTAs are
// persistent over the tiles of their channels.  A gradient comes as its hi and lo parts
// (PARTS = 2, two MMAs per K step).  Every output element sums its taps and channels in the
// same order whatever the plan, so its bits do not depend on it.
//
// Measured on the 16/32/64/128 network at 56 x 56 x 56 voxels, the 14 layers: forward 1158 -> 296 us, data
// gradient 1631 -> 362 us against one voxel row per thread staged anew for each tap (bound by the latency
// of those loads: a coarse layer's 3 or 22 tiles took 27 x 5 us on as many SMs).  At 16 channels a tile now
// costs 2.3 us of an SM for 27 MMAs of 0.02 us: the staging's instructions bound it, which is why small
// plans run with 128 threads (256: 41 us for a 16-channel layer, 128: 23 us); the coarse layers (9 to 36 us)
// are bound by loading up to 390 KB of weights and halo per CTA.
template <int PARTS, typename TO>
__global__ void __launch_bounds__(kConvThreads, 2) k_conv3_tc(Vol g, int K, int N, ConvPlan P, const bf16* __restrict__ in,
                                                           const bf16* __restrict__ in_lo, const bf16* __restrict__ Wrev,
                                                           const float* __restrict__ bias, TO* __restrict__ out,
                                                           int relu, uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bar[kConvStages];
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), threads = blockDim.x;
    const int n0 = blockIdx.y * P.Nc, ahead = ring_ahead(P.stages);
    const uint32_t ncols = tc::tmem_cols(P.Nc);
    if (warp == 0) {
        tc::tmem_alloc(&tbase, ncols);
        tc::tmem_relinquish();
    }
    if (tid == 0)
        for (int i = 0; i < P.stages; ++i) tc::mbar_init(&bar[i], 1);
    const uint32_t sB = tc::smem_u32(smem), sA = sB + (P.resident ? 27u * P.tapB : 0u);
    const int ntx = (g.px + kTx - 1) / kTx, nty = (g.py + kTy - 1) / kTy, nst = 27 / P.taps;
    const int ntiles = ntx * nty * g.pz;
    // weights of `count` taps from `t0`
    auto load_b = [&](int t0, int count, uint32_t dst) {
        const int rows = count * P.Nc;
        for (int e = tid; e < rows * P.kc8; e += threads) {
            const int row = e / P.kc8, c8 = e - row * P.kc8, tt = row / P.Nc, n = row - tt * P.Nc;
            const bool live = n0 + n < N && c8 * 8 < K;
            const bf16* src = live ? Wrev + ((int64_t)(26 - t0 - tt) * N + n0 + n) * K + c8 * 8 : Wrev;
            cp_async16(dst + tt * P.tapB + c8 * P.chunkB + n * 16, src, live);
        }
    };
    // loader state: slot of the ring, stage of the tile, the tile and its first voxel
    const int rowsA = (P.taps == 9 ? kTy + 2 : kTy) * kHx, kcK = K / 8;
    const int step_r = threads / P.kc8, step_c = threads % P.kc8, row0 = tid / P.kc8, col0 = tid % P.kc8;
    int l_slot = 0, l_s = 0, l_tile = blockIdx.x, l_x = 0, l_y = 0, l_z = 0;
    auto load_stage = [&]() {
        if (l_s == 0) {
            const int t = l_tile / ntx;
            l_x = (l_tile - t * ntx) * kTx - 1;
            l_z = t / nty;
            l_y = (t - l_z * nty) * kTy - 1;
        }
        const int s = l_s, z = l_z - 1 + (P.taps == 9 ? s : s / 3), y0 = l_y + (P.taps == 9 ? 0 : s % 3);
        const int64_t base = ((int64_t)l_x + (int64_t)g.px * (y0 + (int64_t)g.py * z)) * K;
        const uint32_t dst = sA + (uint32_t)l_slot * P.stage;
        const unsigned py = z >= 0 && z < g.pz ? (unsigned)g.py : 0u;   // a plane outside the grid: no row is live
        int row = row0, c8 = col0;
        while (row < rowsA) {
            const int yy = row / kHx, xx = row - yy * kHx;
            const bool live = (unsigned)(l_x + xx) < (unsigned)g.px && (unsigned)(y0 + yy) < py && c8 < kcK;
            const int64_t o = live ? base + ((yy * g.px + xx) * K + c8 * 8) : 0;
            const uint32_t d = dst + c8 * P.chunkA + row * 16;
            cp_async16(d, in + o, live);
            if (PARTS == 2) cp_async16(d + P.partA, in_lo + o, live);
            row += step_r;
            c8 += step_c;
            if (c8 >= P.kc8) {
                c8 -= P.kc8;
                ++row;
            }
        }
        if (!P.resident) load_b(s * P.taps, P.taps, dst + PARTS * P.partA);
        if (++l_slot == P.stages) l_slot = 0;
        if (++l_s == nst) {
            l_s = 0;
            l_tile += gridDim.x;
        }
    };
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = tbase;
    const uint32_t idesc = tc::idesc_f16(128, P.Nc, tc::kFmtBF16, 0, 0);
    RingWait ring{bar, P.stages};
    const int total = (int)blockIdx.x < ntiles ? (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * nst : 0;
    bool ok = true;
    if (P.resident) load_b(0, 27, sB);   // arrives with the first stage
    for (int i = 0; i < ahead; ++i) {
        if (i < total) load_stage();
        cp_commit();
    }
    int i = 0, slot = 0, s = 0, tile = blockIdx.x;
    for (; i < total; ++i) {
        if (i + ahead < total) {
            if (i + ahead >= P.stages) ok = ring.upto(i + ahead - P.stages) && ok;
            load_stage();
        }
        cp_commit();
        cp_wait(ahead);
        tc::fence_proxy_async();
        tc::fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
        tc::fence_after_sync();
        if (warp == 0 && tc::elect_one()) {
            const uint32_t a = sA + (uint32_t)slot * P.stage;
            const uint32_t b = P.resident ? sB + (uint32_t)(s * P.taps) * P.tapB : a + PARTS * P.partA;
            uint64_t da = tc::smem_desc(a, P.chunkA, kHx * 16u), db = tc::smem_desc(b, P.chunkB, 128u);
            const uint64_t ka = 2u * P.chunkA >> 4, kb = 2u * P.chunkB >> 4, lo = P.partA >> 4, tb = P.tapB >> 4;
            uint32_t acc = s > 0 ? 1u : 0u;
            auto tap = [&](uint64_t ta) {   // addresses of a descriptor are in units of 16 bytes
                uint64_t td = db;
                for (int k = 0; k < P.kc8; k += 2, ta += ka, td += kb) {
                    tc::mma_f16(taddr, ta, td, idesc, acc);
                    acc = 1u;
                    if (PARTS == 2) tc::mma_f16(taddr, ta + lo, td, idesc, 1u);
                }
                db += tb;
            };
            if (P.taps == 9) {
#pragma unroll
                for (int r = 0; r < 9; ++r) tap(da + (uint64_t)(r / 3 * kHx + r % 3));
            } else {
#pragma unroll
                for (int r = 0; r < 3; ++r) tap(da + (uint64_t)r);
            }
            tc::mma_commit(&bar[slot]);
        }
        __syncwarp();
        if (++slot == P.stages) slot = 0;
        if (++s < nst) continue;
        s = 0;
        ok = ring.upto(i);
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
        tc::fence_after_sync();
        // epilogue: this thread's row, 16 columns at a time, the two halves of the warps in turn
        const int m = tid & 127;
        const int tq = tile / ntx, z = tq / nty;
        const int x = (tile - tq * ntx) * kTx + m % kTx, y = (tq - z * nty) * kTy + m / kTx;
        tile += gridDim.x;
        const bool vin = x < g.px && y < g.py;
        const int64_t v = (int64_t)x + (int64_t)g.px * (y + (int64_t)g.py * z);
        for (int c = 16 * (warp >> 2); c < P.Nc; c += threads >> 3) {
            uint32_t r[16];
            tc::tmem_ld16(tc::tmem_addr(taddr, 32 * (warp & 3), c), r);
            tc::tmem_wait_ld();
            if (!vin) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c0 = n0 + c + 8 * h;
                if (c0 >= N) break;
                float o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float val = __uint_as_float(r[8 * h + j]) + (bias ? bias[c0 + j] : 0.0f);
                    o[j] = relu ? fmaxf(val, 0.0f) : val;
                }
                store8(out + v * N + c0, o);
            }
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
    }
    cp_wait(0);
    if (!ok) {
        if (tid == 0) atomicOr(err, 1u);
        // give MMAs still in flight a bounded time to finish before the TMEM is released
        ring.upto(i - 1, 1u << 16);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(taddr, ncols);
    }
}

// Plan of k_conv3_wgrad_tc.  A CTA owns `taps` taps (27, 9 or 3), `nci` input and `cw` output
// channels: taps * Np accumulator columns, 512 at most.
struct WgradPlan {
    int ty, ntx, nty;    // rows in y of a tile (even), tiles in x and y
    int taps, groups;    // taps of a CTA, groups of taps
    int nci, Np, nchunk; // input channels of a CTA (padded to 16: Np), chunks of them
    int cw, nco;         // output channels of a CTA (64 at most: hi and lo rows make M = 128), chunks of them
    int stages, planes;
    int ntiles, per;     // voxel tiles, tiles per slice
    uint32_t chunkI, planeI, chunkG, stage;
    size_t smem;
};
inline WgradPlan wgrad_plan(const Vol& g, int cin, int cout) {
    WgradPlan p;
    p.ntx = (g.px + kTx - 1) / kTx;
    p.nty = (g.py + kTy - 1) / kTy;
    p.ty = ((g.py + p.nty - 1) / p.nty + 1) / 2 * 2;
    p.ntiles = p.ntx * p.nty * g.pz;
    p.nchunk = cin <= 160 ? 1 : (cin + 127) / 128;
    p.nci = ((cin + p.nchunk - 1) / p.nchunk + 7) / 8 * 8;
    p.Np = (p.nci + 15) / 16 * 16;
    p.taps = 27 * p.Np <= 512 ? 27 : 9 * p.Np <= 512 ? 9 : 3;
    p.groups = 27 / p.taps;
    p.planes = p.taps == 27 ? 3 : 1;
    p.cw = cout < 64 ? cout : 64;
    p.nco = (cout + 63) / 64;
    p.chunkI = (uint32_t)chunk_rows((p.taps == 3 ? p.ty : p.ty + 2) * kHx, p.Np / 8) * 16u;
    p.planeI = (uint32_t)(p.Np / 8) * p.chunkI;
    p.chunkG = (uint32_t)chunk_rows(p.ty * kTx, p.cw / 8) * 16u;
    p.stage = (uint32_t)p.planes * p.planeI + 16u * p.chunkG;
    const int fit = (int)(kSmemOne / p.stage);
    p.stages = fit < kConvStages ? fit : kConvStages;
    p.smem = (size_t)p.stages * p.stage;
    return p;
}

// Weight gradient on the tensor core: part[slice][hi, lo][t][ci][co] = sum over the slice's voxels
// v of in[v + off(t)][ci] g[v][co].  M = 128 rows hold the output channels of the gradient's hi
// part and then of its lo part, N the input channels, one accumulator per tap, K the voxels of a
// tile, two rows in y (16 voxels) per MMA.  Both operands are MN-major: a 16-byte chunk holds 8
// consecutive channels of one voxel, as the channels-last tensors store them; the input of a tap
// is the staged halo at a shifted start address.  Each CTA (grid.y) owns a fixed slice of the
// tiles, and the slices are summed in a fixed order afterwards, so the gradient is deterministic.
// Rows of channels that do not exist multiply whatever the shared memory holds and are not read.
//
// Measured on the same network, the 14 layers: 1981 -> 470 us against rows of (tap, input channel) gathered
// for each group of 128 (27 readings of the input, the gradient split into parts in each).  Bound by the MMA
// count at few channels: 0.03 us per MMA of 128 x 16 x 16, of whose 128 rows 16 output channels use 32.
__global__ void __launch_bounds__(kConvThreads, 2) k_conv3_wgrad_tc(Vol g, int cin, int cout, WgradPlan P,
                                                                 const bf16* __restrict__ in,
                                                                 const bf16* __restrict__ g_hi,
                                                                 const bf16* __restrict__ g_lo,
                                                                 float* __restrict__ part, uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bar[kConvStages];
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), ahead = ring_ahead(P.stages);
    const int grp = blockIdx.x % P.groups, chunk = blockIdx.x / P.groups % P.nchunk;
    const int co0 = blockIdx.x / (P.groups * P.nchunk) * 64, ci0 = chunk * P.nci;
    const int ci1 = ci0 + P.nci < cin ? ci0 + P.nci : cin;
    const uint32_t ncols = tc::tmem_cols(P.taps * P.Np);
    if (warp == 0) {
        tc::tmem_alloc(&tbase, ncols);
        tc::tmem_relinquish();
    }
    if (tid == 0)
        for (int i = 0; i < P.stages; ++i) tc::mbar_init(&bar[i], 1);
    const uint32_t s0 = tc::smem_u32(smem);
    const int first = (int)blockIdx.y * P.per;
    const int total = first + P.per < P.ntiles ? P.per : P.ntiles - first;
    const int kc8 = P.Np / 8, rowsI = (P.taps == 3 ? P.ty : P.ty + 2) * kHx;
    const int gc8 = P.cw / 8, rowsG = P.ty * kTx;
    const int irow = tid / kc8, icol = tid % kc8, istep_r = kConvThreads / kc8, istep_c = kConvThreads % kc8;
    const int grow = tid / gc8, gcol = tid % gc8, gstep_r = kConvThreads / gc8, gstep_c = kConvThreads % gc8;
    const int ilive = (ci1 - ci0) / 8, glive = (cout - co0) / 8;   // chunks that exist
    int l_slot = 0, l_tile = first;
    auto load_stage = [&]() {
        const int tq = l_tile / P.ntx, z0 = tq / P.nty;
        const int x0 = (l_tile - tq * P.ntx) * kTx, y0 = (tq - z0 * P.nty) * P.ty;
        const uint32_t dst = s0 + (uint32_t)l_slot * P.stage;
        const int ya = y0 - 1 + (P.taps == 3 ? grp % 3 : 0);
        for (int pl = 0; pl < P.planes; ++pl) {
            const int z = z0 - 1 + (P.taps == 27 ? pl : P.taps == 9 ? grp : grp / 3);
            const unsigned py = z >= 0 && z < g.pz ? (unsigned)g.py : 0u;   // a plane outside the grid: no row is live
            const int64_t base = ((int64_t)(x0 - 1) + (int64_t)g.px * (ya + (int64_t)g.py * z)) * cin + ci0;
            int row = irow, c8 = icol;
            while (row < rowsI) {
                const int yy = row / kHx, xx = row - yy * kHx;
                const bool live = (unsigned)(x0 - 1 + xx) < (unsigned)g.px && (unsigned)(ya + yy) < py && c8 < ilive;
                const int64_t o = live ? base + ((yy * g.px + xx) * cin + c8 * 8) : 0;
                cp_async16(dst + pl * P.planeI + c8 * P.chunkI + row * 16, in + o, live);
                row += istep_r;
                c8 += istep_c;
                if (c8 >= kc8) {
                    c8 -= kc8;
                    ++row;
                }
            }
        }
        const uint32_t dg = dst + P.planes * P.planeI;
        const int64_t base = ((int64_t)x0 + (int64_t)g.px * (y0 + (int64_t)g.py * z0)) * cout + co0;
        int k = grow, c8 = gcol;
        while (k < rowsG) {
            const int xx = k % kTx, yy = k / kTx;
            const bool live = x0 + xx < g.px && y0 + yy < g.py && c8 < glive;
            const int64_t o = live ? base + ((yy * g.px + xx) * cout + c8 * 8) : 0;
            const uint32_t d = dg + c8 * P.chunkG + k * 16;
            cp_async16(d, g_hi + o, live);
            cp_async16(d + gc8 * P.chunkG, g_lo + o, live);
            k += gstep_r;
            c8 += gstep_c;
            if (c8 >= gc8) {
                c8 -= gc8;
                ++k;
            }
        }
        ++l_tile;
        if (++l_slot == P.stages) l_slot = 0;
    };
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = tbase;
    const uint32_t idesc = tc::idesc_f16(128, P.Np, tc::kFmtBF16, 1, 1);
    RingWait ring{bar, P.stages};
    bool ok = true;
    for (int i = 0; i < ahead; ++i) {
        if (i < total) load_stage();
        cp_commit();
    }
    int i = 0, slot = 0;
    for (; i < total; ++i) {
        if (i + ahead < total) {
            if (i + ahead >= P.stages) ok = ring.upto(i + ahead - P.stages) && ok;
            load_stage();
        }
        cp_commit();
        cp_wait(ahead);
        tc::fence_proxy_async();
        tc::fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
        tc::fence_after_sync();
        if (warp == 0 && tc::elect_one()) {
            const uint32_t a = s0 + (uint32_t)slot * P.stage;
            uint64_t da = tc::smem_desc(a + P.planes * P.planeI, 128u, P.chunkG);
            uint64_t db = tc::smem_desc(a, kHx * 16u, P.chunkI);
            for (int ks = 0; ks < P.ty / 2; ++ks) {   // addresses of a descriptor are in units of 16 bytes
                const uint32_t acc = (i > 0 || ks > 0) ? 1u : 0u;
                uint32_t d = taddr;
                if (P.taps == 3) {
#pragma unroll
                    for (int r = 0; r < 3; ++r, d += P.Np) tc::mma_f16(d, da, db + (uint64_t)r, idesc, acc);
                } else {
                    uint64_t dp = db;
                    for (int pl = 0; pl < P.planes; ++pl, dp += P.planeI >> 4) {
#pragma unroll
                        for (int r = 0; r < 9; ++r, d += P.Np)
                            tc::mma_f16(d, da, dp + (uint64_t)(r / 3 * kHx + r % 3), idesc, acc);
                    }
                }
                da += 16u;
                db += 2u * kHx;
            }
            tc::mma_commit(&bar[slot]);
        }
        __syncwarp();
        if (++slot == P.stages) slot = 0;
    }
    cp_wait(0);
    // every MMA issued (after a failure: bounded time to finish before the TMEM is released)
    ok = ring.upto(i - 1, ok ? 1u << 22 : 1u << 16) && ok;
    ok = __syncthreads_and(ok) != 0;
    tc::fence_after_sync();
    const int m = tid & 127, cwr = gc8 * 8, p = m / cwr, co = co0 + m % cwr;
    for (int c = 16 * (warp >> 2); c < P.taps * P.Np && ok && 32 * (warp & 3) < 2 * cwr; c += 32) {
        uint32_t v[16];
        tc::tmem_ld16(tc::tmem_addr(taddr, 32 * (warp & 3), c), v);
        tc::tmem_wait_ld();
        if (p > 1 || co >= cout) continue;
        const int t = grp * P.taps + c / P.Np, ci = ci0 + c % P.Np;
        float* dst = part + ((((int64_t)blockIdx.y * 2 + p) * 27 + t) * cin + ci) * cout + co;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (ci + j < ci1) dst[(int64_t)j * cout] = __uint_as_float(v[j]);
    }
    if (!ok && tid == 0) atomicOr(err, 1u);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(taddr, ncols);
    }
}

// sum of `slices` values `n` apart, ascending, sixteen loads in flight
__device__ __forceinline__ float ordered_sum(const float* __restrict__ p, int64_t n, int slices) {
    float a = 0.0f;
    int sl = 0;
    for (; sl + 16 <= slices; sl += 16, p += 16 * n) {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = __ldg(p + k * n);
#pragma unroll
        for (int k = 0; k < 16; ++k) a += v[k];
    }
    for (; sl < slices; ++sl, p += n) a += __ldg(p);
    return a;
}
// dst[i] += sum_s part[s][i], s ascending: n1 values of `slices1` slices and behind them n2 of `slices2`
// slices of part2 (a layer's weights and its biases, adjacent in the parameter vector)
__global__ void k_sum_slices(int64_t n1, int slices1, const float* __restrict__ part, int n2, int slices2,
                             const float* __restrict__ part2, float* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n1 + n2) return;
    dst[i] += i < n1 ? ordered_sum(part + i, n1, slices1) : ordered_sum(part2 + (i - n1), n2, slices2);
}

// part[block][co] = sum over the block's voxels of g[v][co] (thread t covers channel t % cout of
// voxels t / cout + k * lanes); the lanes are combined in shared memory in a fixed order
__global__ void k_bias_grad(int64_t nv, int cout, const float* __restrict__ gout, float* __restrict__ part) {
    __shared__ float sp[256];
    const int lanes = blockDim.x / cout;
    const int co = threadIdx.x % cout, sub = threadIdx.x / cout;
    float a = 0.0f;
    for (int64_t v = (int64_t)blockIdx.x * lanes + sub; v < nv; v += (int64_t)gridDim.x * lanes) a += gout[v * cout + co];
    sp[threadIdx.x] = a;
    __syncthreads();
    if (threadIdx.x < cout) {
        float b = 0.0f;
        for (int l = 0; l < lanes; ++l) b += sp[l * cout + threadIdx.x];
        part[(int64_t)blockIdx.x * cout + threadIdx.x] = b;
    }
}

// g = g * (y > 0): gradient through ReLU, y the stored BF16 output of the layer, and the BF16 parts of g for
// the layer's two gradient kernels (split here once: the kernels would split each value per tap and tile);
// eight values per thread, n8 = values / 8
__global__ void k_relu_bwd(int64_t n8, const bf16* __restrict__ y, float* __restrict__ g, bf16* __restrict__ hi,
                           bf16* __restrict__ lo) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n8) return;
    float yv[8], gv[8];
    load8(y + 8 * i, yv);
    load8(g + 8 * i, gv);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (!(yv[k] > 0.0f)) gv[k] = 0.0f;
    store8(g + 8 * i, gv);
    uint4 h, l;
    split8(gv, h, l);
    reinterpret_cast<uint4*>(hi)[i] = h;
    reinterpret_cast<uint4*>(lo)[i] = l;
}

// 2x2x2 average pooling (fine -> coarse), BF16
__global__ void k_pool(Vol f, Vol c, int ch, const bf16* __restrict__ in, bf16* __restrict__ out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nv * ch) return;
    const int64_t V = i / ch;
    const int cc = (int)(i % ch);
    const int X = (int)(V % c.px), Y = (int)((V / c.px) % c.py), Z = (int)(V / ((int64_t)c.px * c.py));
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = 2 * X + (k & 1), y = 2 * Y + ((k >> 1) & 1), z = 2 * Z + (k >> 2);
        s += __bfloat162float(in[((int64_t)x + (int64_t)f.px * (y + (int64_t)f.py * z)) * ch + cc]);
    }
    out[i] = __float2bfloat16_rn(0.125f * s);
}

// gradient of the pooling, added: gf[v][c] += gc[parent(v)][c] / 8
__global__ void k_pool_bwd_add(Vol f, Vol c, int ch, const float* __restrict__ gc, float* __restrict__ gf) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= f.nv * ch) return;
    const int64_t v = i / ch;
    const int cc = (int)(i % ch);
    const int x = (int)(v % f.px), y = (int)((v / f.px) % f.py), z = (int)(v / ((int64_t)f.px * f.py));
    const int64_t V = (x / 2) + (int64_t)c.px * ((y / 2) + (int64_t)c.py * (z / 2));
    gf[i] += 0.125f * gc[V * ch + cc];
}

// decoder input: out[v] = [ up(coarse)[v] (cu channels) | skip[v] (cs channels) ], eight channels per thread
__global__ void k_up_concat(Vol f, Vol c, int cu, int cs, const bf16* __restrict__ coarse,
                            const bf16* __restrict__ skip, bf16* __restrict__ out) {
    const int ct8 = (cu + cs) / 8;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= f.nv * ct8) return;
    const int64_t v = i / ct8;
    const int cc = (int)(i - v * ct8) * 8;
    const bf16* src;
    if (cc < cu) {
        const int64_t row = v / f.px;
        const int x = (int)(v - row * f.px), z = (int)(row / f.py), y = (int)(row - (int64_t)z * f.py);
        const int64_t V = (x / 2) + (int64_t)c.px * ((y / 2) + (int64_t)c.py * (z / 2));
        src = coarse + V * cu + cc;
    } else {
        src = skip + v * cs + (cc - cu);
    }
    reinterpret_cast<uint4*>(out)[i] = __ldg(reinterpret_cast<const uint4*>(src));
}

// gradient of k_up_concat: gc[V][c] = sum over the 8 children of g[v][c] (c < cu);
// gskip[v][c] += g[v][cu + c]
__global__ void k_up_concat_bwd_coarse(Vol f, Vol c, int cu, int cs, const float* __restrict__ g,
                                       float* __restrict__ gc) {
    const int ct = cu + cs;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nv * cu) return;
    const int64_t V = i / cu;
    const int cc = (int)(i % cu);
    const int X = (int)(V % c.px), Y = (int)((V / c.px) % c.py), Z = (int)(V / ((int64_t)c.px * c.py));
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = 2 * X + (k & 1), y = 2 * Y + ((k >> 1) & 1), z = 2 * Z + (k >> 2);
        s += g[((int64_t)x + (int64_t)f.px * (y + (int64_t)f.py * z)) * ct + cc];
    }
    gc[i] = s;
}
__global__ void k_up_concat_bwd_skip(Vol f, int cu, int cs, const float* __restrict__ g, float* __restrict__ gs) {
    const int ct = cu + cs;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= f.nv * cs) return;
    const int64_t v = i / cs;
    const int cc = (int)(i % cs);
    gs[i] += g[v * ct + cu + cc];
}

// head: out[d][v] = b[d] + sum_c W[c][d] x[v][c]   (d < 3, out SoA FP32)
__global__ void k_head(int64_t nv, int cin, const bf16* __restrict__ x, const float* __restrict__ W,
                       const float* __restrict__ b, float* __restrict__ out) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    float a0 = b[0], a1 = b[1], a2 = b[2];
    for (int c8 = 0; c8 < cin; c8 += 8) {
        float xv[8];
        load8(x + v * cin + c8, xv);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float* w = W + (c8 + c) * 3;
            a0 = fmaf(xv[c], w[0], a0);
            a1 = fmaf(xv[c], w[1], a1);
            a2 = fmaf(xv[c], w[2], a2);
        }
    }
    out[v] = a0;
    out[nv + v] = a1;
    out[2 * nv + v] = a2;
}

// head backward: gx[v][c] = sum_d W[c][d] g[d][v]; dW[c][d] += sum_v x[v][c] g[d][v]; db[d] += sum_v g[d][v]
// (warp sums first, then one shared-memory add per warp, then one global add per block)
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// part[block][0 .. 3 cin) = block sums of x[v][c] g[d][v], part[block][3 cin .. 3 cin + 3) = of g[d][v]
// (warp sums, then the warps in a fixed order); gx[v][c] = sum_d W[c][d] g[d][v]
__global__ void k_head_bwd(int64_t nv, int cin, const bf16* __restrict__ x, const float* __restrict__ W,
                           const float* __restrict__ g, float* __restrict__ gx, float* __restrict__ part) {
    extern __shared__ float swarp[];   // [warps][cin * 3 + 3]
    const int nq = cin * 3 + 3, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool act = v < nv;
    const float g0 = act ? g[v] : 0.0f, g1 = act ? g[nv + v] : 0.0f, g2 = act ? g[2 * nv + v] : 0.0f;
    const bool lead = (threadIdx.x & 31) == 0;
    for (int c = 0; c < cin; ++c) {
        const float* w = W + c * 3;
        const float xv = act ? __bfloat162float(x[v * cin + c]) : 0.0f;
        if (act) gx[v * cin + c] = w[0] * g0 + w[1] * g1 + w[2] * g2;
        const float s0 = warp_sum(xv * g0), s1 = warp_sum(xv * g1), s2 = warp_sum(xv * g2);
        if (lead) {
            swarp[warp * nq + c * 3 + 0] = s0;
            swarp[warp * nq + c * 3 + 1] = s1;
            swarp[warp * nq + c * 3 + 2] = s2;
        }
    }
    const float t0 = warp_sum(g0), t1 = warp_sum(g1), t2 = warp_sum(g2);
    if (lead) {
        swarp[warp * nq + cin * 3 + 0] = t0;
        swarp[warp * nq + cin * 3 + 1] = t1;
        swarp[warp * nq + cin * 3 + 2] = t2;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nq; k += blockDim.x) {
        float a = 0.0f;
        for (int w = 0; w < nw; ++w) a += swarp[w * nq + k];
        part[(int64_t)blockIdx.x * nq + k] = a;
    }
}

// FP32 master weights -> BF16 W[t][ci][co] and the flipped transpose W'[t][co][ci] = W[26-t][ci][co]
__global__ void k_pack(int taps, int cin, int cout, const float* __restrict__ w, bf16* __restrict__ w16,
                       bf16* __restrict__ wflip) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = (int64_t)taps * cin * cout;
    if (i >= n) return;
    const int t = (int)(i / ((int64_t)cin * cout));
    const int rem = (int)(i % ((int64_t)cin * cout));
    const int ci = rem / cout, co = rem % cout;
    const bf16 b = __float2bfloat16_rn(w[i]);
    w16[i] = b;
    if (wflip) wflip[((int64_t)(taps - 1 - t) * cout + co) * cin + ci] = b;
}

// Adam (Kingma & Ba 2015) with bias correction; bc1 = 1 - beta1^t, bc2 = 1 - beta2^t
__global__ void k_adam(int64_t n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float bc1, float bc2,
                       float gscale) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] * gscale;
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
static unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

static int sm_count(Context& c) {
    int n = 0;
    UWG_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, c.device));
    return n > 0 ? n : 1;
}

void check_errors(Context& c, Net& n) {
    if (!n.tc_err.p) return;
    uint32_t e = 0;
    UWG_CUDA(cudaMemcpyAsync(&e, n.tc_err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    if (e) {
        UWG_CUDA(cudaMemsetAsync(n.tc_err.p, 0, sizeof(uint32_t), c.stream));
        throw Error(UWGPU_ERR_CUDA, "U-Net tensor-core kernel: an MMA did not complete in time");
    }
}

// 3x3x3 convolution on the tensor core (k_conv3_tc).  Wrev: the layer's packing with the output channel
// before the input channel, [27][N][K] in reverse tap order.  The widths accepted are those of which one
// tap's weights and 128 voxels' inputs fit a CTA's shared memory twice.
template <int PARTS, typename TO>
static void conv_launch_tc(Context& c, Net& n, const Vol& g, int K, int N, const bf16* in, const bf16* in_lo,
                           const bf16* Wrev, const float* bias, TO* out, bool relu) {
    const int Kp = (K + 15) / 16 * 16, Np = (N + 15) / 16 * 16;
    UWG_REQUIRE(Np <= 256, UWGPU_ERR_ARGUMENT, "U-Net layer too wide for the tensor-core convolution");
    UWG_REQUIRE((size_t)4 * Kp * (Np + PARTS * 128) <= kSmemWidth, UWGPU_ERR_ARGUMENT,
                "tensor-core kernel: shared memory plan too large");
    const int64_t ntiles = (int64_t)((g.px + kTx - 1) / kTx) * ((g.py + kTy - 1) / kTy) * g.pz;
    const int sms = sm_count(c);
    const ConvPlan P = conv_plan(K, N, PARTS, ntiles, sms);
    int per_sm = 1;
    const size_t smem =
        tmem_safe_smem((const void*)k_conv3_tc<PARTS, TO>, c.device, P.smem, tc::tmem_cols(P.Nc), &per_sm);
    const int threads = P.smem <= kSmemTwo ? 128 : kConvThreads;
    if (per_sm > 2048 / threads) per_sm = 2048 / threads;
    const int64_t cap = std::max<int64_t>((int64_t)sms * per_sm / P.nchunks, 1);
    const dim3 grid((unsigned)(ntiles < cap ? ntiles : cap), (unsigned)P.nchunks);
    LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
    k_conv3_tc<PARTS, TO><<<grid, threads, smem, c.stream>>>(g, K, N, P, in, in_lo, Wrev, bias, out, relu ? 1 : 0,
                                                                  n.tc_err.p);
    note_work(c, UWGPU_KERNEL_LEARNED, (double)g.nv * (K * PARTS * sizeof(bf16) + N * sizeof(TO)),
              2.0 * 27.0 * K * N * (double)g.nv * PARTS);
}

// dW += the weight gradient from the layer's input and the parts (n.g_hi, n.g_lo) of its output gradient
// gout; db (behind dW in the parameter vector) += the sums of gout
static void wgrad_launch_tc(Context& c, Net& n, const Vol& g, int cin, int cout, const bf16* in, const float* gout,
                            float* dW, DArray<float>& part) {
    constexpr int kBiasBlocks = 152;
    UWG_REQUIRE(cout <= 256, UWGPU_ERR_ARGUMENT, "U-Net layer too wide for the tensor-core weight gradient");
    WgradPlan P = wgrad_plan(g, cin, cout);
    int per_sm = 1;
    const size_t smem =
        tmem_safe_smem((const void*)k_conv3_wgrad_tc, c.device, P.smem, tc::tmem_cols(P.taps * P.Np), &per_sm);
    const int gx = P.groups * P.nchunk * P.nco;
    int slices = std::max(sm_count(c) * per_sm / gx, 1);
    if (slices > P.ntiles) slices = P.ntiles;
    P.per = (P.ntiles + slices - 1) / slices;
    slices = (P.ntiles + P.per - 1) / P.per;
    const int64_t nw = (int64_t)27 * cin * cout;
    part.ensure((size_t)slices * 2 * nw + (size_t)kBiasBlocks * cout);
    float* bias_part = part.p + (size_t)slices * 2 * nw;
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_bias_grad<<<kBiasBlocks, (256 / cout) * cout, 0, c.stream>>>(g.nv, cout, gout, bias_part);
    }
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_conv3_wgrad_tc<<<dim3(gx, (unsigned)slices), kConvThreads, smem, c.stream>>>(g, cin, cout, P, in, n.g_hi.p,
                                                                                      n.g_lo.p, part.p, n.tc_err.p);
    }
    LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
    k_sum_slices<<<nblk(nw + cout, 256), 256, 0, c.stream>>>(nw, 2 * slices, part.p, cout, kBiasBlocks, bias_part, dW);
    note_work(c, UWGPU_KERNEL_LEARNED, (double)g.nv * 27.0 * (cin * 2 + cout * 4), 4.0 * 27.0 * cin * cout * (double)g.nv);
}

static void relu_bwd(Context& c, Net& n, int64_t count, const bf16* y, float* g) {
    LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
    k_relu_bwd<<<nblk(count / 8, 256), 256, 0, c.stream>>>(count / 8, y, g, n.g_hi.p, n.g_lo.p);
}

// splitmix64 (Steele, Lea and Flood 2014) for reproducible initial weights
static uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

void destroy(Net* n) { delete n; }

void create(Context& c, Net& n, int levels, int base, uint64_t seed) {
    const MeshDesc& m = c.mesh;
    UWG_REQUIRE(m.dim == 3, UWGPU_ERR_UNSUPPORTED, "the learned preconditioner is built for 3D meshes");
    UWG_REQUIRE(levels >= 1 && levels <= kMaxLevels, UWGPU_ERR_ARGUMENT, "U-Net levels must be 1..6");
    UWG_REQUIRE(base >= 8 && base % 8 == 0 && (base << (levels - 1)) <= 256, UWGPU_ERR_ARGUMENT,
                "U-Net base channels must be a multiple of 8, at most 256 at the coarsest level");
    n.levels = levels;
    n.base = base;
    n.nnx = m.nnx;
    n.nny = m.nny;
    n.nnz = m.nnz;
    n.nn = m.nn;
    const int64_t mult = (int64_t)1 << (levels - 1);
    Vol v0;
    v0.px = (int)((m.nnx + mult - 1) / mult * mult);
    v0.py = (int)((m.nny + mult - 1) / mult * mult);
    v0.pz = (int)((m.nnz + mult - 1) / mult * mult);
    for (int l = 0; l < levels; ++l) {
        Vol v;
        v.px = v0.px >> l;
        v.py = v0.py >> l;
        v.pz = v0.pz >> l;
        v.nv = (int64_t)v.px * v.py * v.pz;
        n.vol[l] = v;
        n.ch[l] = base << l;
    }
    // layers and parameter offsets
    {
        std::vector<Conv> fresh((size_t)(2 * levels + 2 * (levels - 1)));   // Conv owns device arrays: no copies
        n.convs.swap(fresh);
    }
    int64_t off = 0;
    auto add = [&](Conv& cv, int cin, int cout) {
        cv.cin = cin;
        cv.cout = cout;
        cv.w_off = off;
        off += (int64_t)27 * cin * cout;
        cv.b_off = off;
        off += cout;
    };
    for (int l = 0; l < levels; ++l) {
        add(n.convs[n.enc(l, 0)], n.cin_of_level(l), n.ch[l]);
        add(n.convs[n.enc(l, 1)], n.ch[l], n.ch[l]);
    }
    for (int l = 0; l + 1 < levels; ++l) {
        add(n.convs[n.dec(l, 0)], n.ch[l + 1] + n.ch[l], n.ch[l]);
        add(n.convs[n.dec(l, 1)], n.ch[l], n.ch[l]);
    }
    n.head_w = off;
    off += (int64_t)n.ch[0] * 3;
    n.head_b = off;
    off += 3;
    n.nparams = off;
    // He-uniform initial weights, zero biases, zero head (the untrained net adds nothing)
    std::vector<float> h((size_t)n.nparams, 0.0f);
    uint64_t s = seed;
    for (auto& cv : n.convs) {
        const float a = std::sqrt(6.0f / (27.0f * cv.cin));
        for (int64_t i = 0; i < (int64_t)27 * cv.cin * cv.cout; ++i) {
            const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
            h[(size_t)(cv.w_off + i)] = (float)((2.0 * u - 1.0) * a);
        }
    }
    for (auto* a : {&n.params, &n.grads, &n.adam_m, &n.adam_v}) a->ensure((size_t)n.nparams);
    UWG_CUDA(cudaMemcpy(n.params.p, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
    UWG_CUDA(cudaMemset(n.grads.p, 0, h.size() * sizeof(float)));
    UWG_CUDA(cudaMemset(n.adam_m.p, 0, h.size() * sizeof(float)));
    UWG_CUDA(cudaMemset(n.adam_v.p, 0, h.size() * sizeof(float)));
    n.adam_t = 0;
    n.out_scale = 1.0f;
    // activations and gradients
    const Vol& f = n.vol[0];
    n.x0.ensure((size_t)f.nv * kInChannels);
    UWG_CUDA(cudaMemset(n.x0.p, 0, (size_t)f.nv * kInChannels * sizeof(bf16)));
    n.out.ensure((size_t)f.nv * 3);
    n.gout.ensure((size_t)f.nv * 3);
    for (int l = 0; l < levels; ++l) {
        const int64_t nv = n.vol[l].nv;
        const int C = n.ch[l];
        n.g_hi.ensure((size_t)nv * C);
        n.g_lo.ensure((size_t)nv * C);
        n.enc_a[l].ensure((size_t)nv * C);
        n.enc_b[l].ensure((size_t)nv * C);
        n.g_enc_a[l].ensure((size_t)nv * C);
        n.g_enc_b[l].ensure((size_t)nv * C);
        n.g_in[l].ensure((size_t)nv * n.cin_of_level(l));
        if (l + 1 < levels) {
            n.pool[l].ensure((size_t)n.vol[l + 1].nv * C);
            const int ct = n.ch[l + 1] + C;
            n.dec_cat[l].ensure((size_t)nv * ct);
            n.dec_a[l].ensure((size_t)nv * C);
            n.dec_b[l].ensure((size_t)nv * C);
            n.g_cat[l].ensure((size_t)nv * ct);
            n.g_dec_a[l].ensure((size_t)nv * C);
            n.g_dec_b[l].ensure((size_t)nv * C);
        }
    }
    for (auto& cv : n.convs) {
        cv.w16.ensure((size_t)27 * cv.cin * cv.cout);
        cv.wflip.ensure((size_t)27 * cv.cin * cv.cout);
    }
    n.tc_err.ensure(1);
    UWG_CUDA(cudaMemset(n.tc_err.p, 0, sizeof(uint32_t)));
    pack(c, n);
}

void pack(Context& c, Net& n) {
    for (auto& cv : n.convs) {
        const int64_t nw = (int64_t)27 * cv.cin * cv.cout;
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_pack<<<nblk(nw, 256), 256, 0, c.stream>>>(27, cv.cin, cv.cout, n.params.p + cv.w_off, cv.w16.p, cv.wflip.p);
    }
    check_launch("k_pack");
}

void forward(Context& c, Net& n) {
    const int L = n.levels;
    for (int l = 0; l < L; ++l) {
        const Vol& g = n.vol[l];
        const Conv& a = n.convs[n.enc(l, 0)];
        const Conv& b = n.convs[n.enc(l, 1)];
        const bf16* in = l == 0 ? n.x0.p : n.pool[l - 1].p;
        conv_launch_tc<1, bf16>(c, n, g, a.cin, a.cout, in, nullptr, a.wflip.p, n.params.p + a.b_off, n.enc_a[l].p, true);
        conv_launch_tc<1, bf16>(c, n, g, b.cin, b.cout, n.enc_a[l].p, nullptr, b.wflip.p, n.params.p + b.b_off,
                                n.enc_b[l].p, true);
        if (l + 1 < L) {
            const int64_t cnt = n.vol[l + 1].nv * n.ch[l];
            LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
            k_pool<<<nblk(cnt, 256), 256, 0, c.stream>>>(g, n.vol[l + 1], n.ch[l], n.enc_b[l].p, n.pool[l].p);
        }
    }
    for (int l = L - 2; l >= 0; --l) {
        const Vol& g = n.vol[l];
        const int cu = n.ch[l + 1], cs = n.ch[l];
        const bf16* coarse = l == L - 2 ? n.enc_b[L - 1].p : n.dec_b[l + 1].p;
        {
            const int64_t cnt = g.nv * ((cu + cs) / 8);
            LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
            k_up_concat<<<nblk(cnt, 256), 256, 0, c.stream>>>(g, n.vol[l + 1], cu, cs, coarse, n.enc_b[l].p,
                                                              n.dec_cat[l].p);
        }
        const Conv& a = n.convs[n.dec(l, 0)];
        const Conv& b = n.convs[n.dec(l, 1)];
        conv_launch_tc<1, bf16>(c, n, g, a.cin, a.cout, n.dec_cat[l].p, nullptr, a.wflip.p, n.params.p + a.b_off,
                                n.dec_a[l].p, true);
        conv_launch_tc<1, bf16>(c, n, g, b.cin, b.cout, n.dec_a[l].p, nullptr, b.wflip.p, n.params.p + b.b_off,
                                n.dec_b[l].p, true);
    }
    const bf16* fin = L == 1 ? n.enc_b[0].p : n.dec_b[0].p;
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_head<<<nblk(n.vol[0].nv, 256), 256, 0, c.stream>>>(n.vol[0].nv, n.ch[0], fin, n.params.p + n.head_w,
                                                              n.params.p + n.head_b, n.out.p);
    }
    check_launch("unet forward");
}

// gradient of one conv layer: g (pre-activation gradient, FP32, [nv][cout], its parts in n.g_hi and n.g_lo)
// -> dW, db, and the gradient of its input (post-activation of the layer below) into gin
static void conv_backward(Context& c, Net& n, const Vol& g, const Conv& cv, const bf16* in, const float* gpre,
                          float* gin) {
    wgrad_launch_tc(c, n, g, cv.cin, cv.cout, in, gpre, n.grads.p + cv.w_off, n.part);
    // the data gradient is the convolution with W'[t][co][ci] = W[26 - t][ci][co]; its other
    // packing, read in reverse tap order, is the plain W
    conv_launch_tc<2, float>(c, n, g, cv.cout, cv.cin, n.g_hi.p, n.g_lo.p, cv.w16.p, nullptr, gin, false);
}

void backward(Context& c, Net& n) {
    const int L = n.levels;
    const Vol& f = n.vol[0];
    const bf16* fin = L == 1 ? n.enc_b[0].p : n.dec_b[0].p;
    float* gfin = L == 1 ? n.g_enc_b[0].p : n.g_dec_b[0].p;
    {
        const int nq = n.ch[0] * 3 + 3;
        const unsigned hb = nblk(f.nv, 256);
        n.part.ensure((size_t)hb * nq);
        {
            LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
            k_head_bwd<<<hb, 256, (size_t)8 * nq * sizeof(float), c.stream>>>(f.nv, n.ch[0], fin, n.params.p + n.head_w,
                                                                              n.gout.p, gfin, n.part.p);
        }
        // head_w and head_b are adjacent in the parameter vector: one ordered sum for both
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_sum_slices<<<nblk(nq, 256), 256, 0, c.stream>>>(nq, (int)hb, n.part.p, 0, 0, nullptr, n.grads.p + n.head_w);
    }
    // skip gradients start at zero; the decoder adds into them
    for (int l = 0; l + 1 < L; ++l)
        UWG_CUDA(cudaMemsetAsync(n.g_enc_b[l].p, 0, (size_t)n.vol[l].nv * n.ch[l] * sizeof(float), c.stream));
    for (int l = 0; l + 1 < L; ++l) {
        const Vol& g = n.vol[l];
        const int cu = n.ch[l + 1], cs = n.ch[l];
        relu_bwd(c, n, g.nv * cs, n.dec_b[l].p, n.g_dec_b[l].p);
        conv_backward(c, n, g, n.convs[n.dec(l, 1)], n.dec_a[l].p, n.g_dec_b[l].p, n.g_dec_a[l].p);
        relu_bwd(c, n, g.nv * cs, n.dec_a[l].p, n.g_dec_a[l].p);
        conv_backward(c, n, g, n.convs[n.dec(l, 0)], n.dec_cat[l].p, n.g_dec_a[l].p, n.g_cat[l].p);
        float* gcoarse = l + 1 == L - 1 ? n.g_enc_b[L - 1].p : n.g_dec_b[l + 1].p;
        {
            LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
            k_up_concat_bwd_coarse<<<nblk(n.vol[l + 1].nv * cu, 256), 256, 0, c.stream>>>(g, n.vol[l + 1], cu, cs,
                                                                                           n.g_cat[l].p, gcoarse);
        }
        {
            LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
            k_up_concat_bwd_skip<<<nblk(g.nv * cs, 256), 256, 0, c.stream>>>(g, cu, cs, n.g_cat[l].p, n.g_enc_b[l].p);
        }
    }
    for (int l = L - 1; l >= 0; --l) {
        const Vol& g = n.vol[l];
        const int C = n.ch[l];
        if (l + 1 < L) {
            LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
            k_pool_bwd_add<<<nblk(g.nv * C, 256), 256, 0, c.stream>>>(g, n.vol[l + 1], C, n.g_in[l + 1].p,
                                                                      n.g_enc_b[l].p);
        }
        relu_bwd(c, n, g.nv * C, n.enc_b[l].p, n.g_enc_b[l].p);
        conv_backward(c, n, g, n.convs[n.enc(l, 1)], n.enc_a[l].p, n.g_enc_b[l].p, n.g_enc_a[l].p);
        relu_bwd(c, n, g.nv * C, n.enc_a[l].p, n.g_enc_a[l].p);
        const bf16* in = l == 0 ? n.x0.p : n.pool[l - 1].p;
        conv_backward(c, n, g, n.convs[n.enc(l, 0)], in, n.g_enc_a[l].p, n.g_in[l].p);
    }
    check_launch("unet backward");
}

// node (i, j, k) of the mesh sits at voxel (i, j, k) of the padded level-0 grid
__global__ void k_input_from_host_layout(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ in4,
                                         bf16* __restrict__ x0) {
    int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t i = node % nnx, j = (node / nnx) % nny, k = node / (nnx * nny);
    const int64_t v = i + (int64_t)g.px * (j + (int64_t)g.py * k);
#pragma unroll
    for (int ch = 0; ch < kUsedChannels; ++ch) x0[v * kInChannels + ch] = __float2bfloat16_rn(in4[(int64_t)ch * nn + node]);
}

__global__ void k_output_to_node_layout(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ out,
                                        float* __restrict__ o3) {
    int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t i = node % nnx, j = (node / nnx) % nny, k = node / (nnx * nny);
    const int64_t v = i + (int64_t)g.px * (j + (int64_t)g.py * k);
#pragma unroll
    for (int d = 0; d < 3; ++d) o3[(int64_t)d * nn + node] = out[(int64_t)d * g.nv + v];
}

void set_input_host(Context& c, Net& n, const float* input) {
    DArray<float> tmp;
    tmp.ensure((size_t)n.nn * kUsedChannels);
    UWG_CUDA(cudaMemcpyAsync(tmp.p, input, (size_t)n.nn * kUsedChannels * sizeof(float), cudaMemcpyHostToDevice,
                             c.stream));
    UWG_CUDA(cudaMemsetAsync(n.x0.p, 0, (size_t)n.vol[0].nv * kInChannels * sizeof(bf16), c.stream));
    LaunchScope ls(c, -1);
    k_input_from_host_layout<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], tmp.p, n.x0.p);
    UWG_CUDA(cudaStreamSynchronize(c.stream));
}

void get_output_host(Context& c, Net& n, float* output) {
    check_errors(c, n);
    DArray<float> tmp;
    tmp.ensure((size_t)n.nn * 3);
    {
        LaunchScope ls(c, -1);
        k_output_to_node_layout<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], n.out.p, tmp.p);
    }
    UWG_CUDA(cudaMemcpyAsync(output, tmp.p, (size_t)n.nn * 3 * sizeof(float), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
}

__global__ void k_grad_from_node_layout(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ g3,
                                        float* __restrict__ gout) {
    int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t i = node % nnx, j = (node / nnx) % nny, k = node / (nnx * nny);
    const int64_t v = i + (int64_t)g.px * (j + (int64_t)g.py * k);
#pragma unroll
    for (int d = 0; d < 3; ++d) gout[(int64_t)d * g.nv + v] = g3[(int64_t)d * nn + node];
}

__global__ void k_input_grad_to_node_layout(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ gin,
                                            float* __restrict__ g4) {
    int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t i = node % nnx, j = (node / nnx) % nny, k = node / (nnx * nny);
    const int64_t v = i + (int64_t)g.px * (j + (int64_t)g.py * k);
#pragma unroll
    for (int ch = 0; ch < kUsedChannels; ++ch) g4[(int64_t)ch * nn + node] = gin[v * kInChannels + ch];
}

void set_grad_output_host(Context& c, Net& n, const float* grad) {
    DArray<float> tmp;
    tmp.ensure((size_t)n.nn * 3);
    UWG_CUDA(cudaMemcpyAsync(tmp.p, grad, (size_t)n.nn * 3 * sizeof(float), cudaMemcpyHostToDevice, c.stream));
    UWG_CUDA(cudaMemsetAsync(n.gout.p, 0, (size_t)n.vol[0].nv * 3 * sizeof(float), c.stream));
    LaunchScope ls(c, -1);
    k_grad_from_node_layout<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], tmp.p, n.gout.p);
    UWG_CUDA(cudaStreamSynchronize(c.stream));
}

void get_input_grad_host(Context& c, Net& n, float* grad_input) {
    check_errors(c, n);
    DArray<float> tmp;
    tmp.ensure((size_t)n.nn * kUsedChannels);
    {
        LaunchScope ls(c, -1);
        k_input_grad_to_node_layout<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], n.g_in[0].p,
                                                                            tmp.p);
    }
    UWG_CUDA(cudaMemcpyAsync(grad_input, tmp.p, (size_t)n.nn * kUsedChannels * sizeof(float), cudaMemcpyDeviceToHost,
                             c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
}

// ------------------------------------------------------------------------------------------
// The network as a preconditioner: residual -> input tensor, output -> velocity correction
// ------------------------------------------------------------------------------------------
// out[0] += sum x^2, in a fixed order: launched as one block of 1024 threads (deterministic)
template <typename T>
__global__ void __launch_bounds__(1024) k_sumsq(int64_t n, const T* __restrict__ x, double* __restrict__ out) {
    __shared__ double sw[32];
    float sf = 0.0f;   // each thread's strided partial in FP32 (fixed order), the tree in FP64
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const float v = (float)x[i];
        sf = fmaf(v, v, sf);
    }
    double s = sf;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sw[w];
        out[0] += t;
    }
}

// node (i, j, k) of the mesh is voxel (i, j, k) of the padded level-0 grid
__device__ __forceinline__ int64_t node_voxel(int64_t node, int64_t nnx, int64_t nny, const Vol& g) {
    const int64_t i = node % nnx, j = (node / nnx) % nny, k = node / (nnx * nny);
    return i + (int64_t)g.px * (j + (int64_t)g.py * k);
}

// x0[v] = (r / rms(r), v / rms(v), log10 viscosity, 0) at node voxels; sumsq = (|r|^2, |v|^2)
template <typename T>
__global__ void k_make_input(int64_t nnx, int64_t nny, int64_t nn, Vol g, const T* __restrict__ r,
                             const T* __restrict__ vc, const double* __restrict__ sumsq,
                             const float* __restrict__ logeta, bf16* __restrict__ x0) {
    __shared__ float inv[2];
    if (threadIdx.x < 2)
        inv[threadIdx.x] = sumsq[threadIdx.x] > 0.0 ? (float)rsqrt(sumsq[threadIdx.x] / (double)(3 * nn)) : 0.0f;
    __syncthreads();
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t v = node_voxel(node, nnx, nny, g);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        x0[v * kInChannels + d] = __float2bfloat16_rn((float)r[(int64_t)d * nn + node] * inv[0]);
        x0[v * kInChannels + 3 + d] = __float2bfloat16_rn((float)vc[(int64_t)d * nn + node] * inv[1]);
    }
    x0[v * kInChannels + 6] = __float2bfloat16_rn(logeta[node]);
}

// z[d][node] += out_scale * rms(V(r)) * out[d][v] on free dofs (sumsq[1] = |V(r)|^2)
template <typename T>
__global__ void k_add_correction(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ out,
                                 const double* __restrict__ sumsq, float out_scale, const uint8_t* __restrict__ fixed,
                                 T* __restrict__ z) {
    __shared__ float s;
    if (threadIdx.x == 0) s = out_scale * (float)sqrt(sumsq[1] / (double)(3 * nn));
    __syncthreads();
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t v = node_voxel(node, nnx, nny, g);
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (!(fixed && fixed[node * 3 + d])) z[(int64_t)d * nn + node] += (T)(s * out[(int64_t)d * g.nv + v]);
}

// mean of log10(viscosity) over the material points of each element (0 for an empty element)
__global__ void k_elem_logeta(int64_t ne, const uint32_t* __restrict__ offsets, const double* __restrict__ eta,
                              float* __restrict__ elog) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const uint32_t a = offsets[e], b = offsets[e + 1];
    float s = 0.0f;
    for (uint32_t k = a; k < b; ++k) s += log10f(fmaxf((float)eta[k], 1e-30f));
    elog[e] = b > a ? s / (float)(b - a) : 0.0f;
}

// node value = mean over the (1..8) elements around the node
__global__ void k_node_logeta(int64_t nnx, int64_t nny, int64_t nn, int ex, int ey, int ez, const float* __restrict__ elog,
                              float* __restrict__ nlog) {
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t i = node % nnx, j = (node / nnx) % nny, k = node / (nnx * nny);
    float s = 0.0f;
    int cnt = 0;
    for (int o = 0; o < 8; ++o) {
        const int64_t a = i - (o & 1), b = j - ((o >> 1) & 1), cc = k - (o >> 2);
        if (a < 0 || a >= ex || b < 0 || b >= ey || cc < 0 || cc >= ez) continue;
        s += elog[a + (int64_t)ex * (b + (int64_t)ey * cc)];
        cnt++;
    }
    nlog[node] = cnt ? s / (float)cnt : 0.0f;
}

void prepare_viscosity(Context& c, Net& n) {
    UWG_REQUIRE(c.assembled && c.mapped, UWGPU_ERR_STATE, "learned preconditioner needs the assembled point viscosities");
    const MeshDesc& m = c.mesh;
    n.logeta.ensure((size_t)n.nn);
    DArray<float> elog;
    elog.ensure((size_t)m.ne);
    {
        LaunchScope ls(c, -1);
        k_elem_logeta<<<nblk(m.ne, 256), 256, 0, c.stream>>>(m.ne, c.offsets.p, c.seta_out.p, elog.p);
    }
    {
        LaunchScope ls(c, -1);
        k_node_logeta<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, m.nel[0], m.nel[1], m.nel[2], elog.p,
                                                             n.logeta.p);
    }
    UWG_CUDA(cudaStreamSynchronize(c.stream));   // elog is released on return
}

template <typename T>
void correct(Context& c, Net& n, const T* r, T* z) {
    n.sumsq.ensure(2);
    UWG_CUDA(cudaMemsetAsync(n.sumsq.p, 0, 2 * sizeof(double), c.stream));
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_sumsq<T><<<1, 1024, 0, c.stream>>>(3 * n.nn, r, n.sumsq.p);
    }
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_sumsq<T><<<1, 1024, 0, c.stream>>>(3 * n.nn, z, n.sumsq.p + 1);
    }
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_make_input<T><<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], r, z, n.sumsq.p,
                                                                n.logeta.p, n.x0.p);
    }
    forward(c, n);
    LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
    k_add_correction<T><<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], n.out.p, n.sumsq.p,
                                                                n.out_scale, c.levels[0].fixed.p, z);
}
template void correct<double>(Context&, Net&, const double*, double*);
template void correct<float>(Context&, Net&, const float*, float*);

// ------------------------------------------------------------------------------------------
// Training data: residual/error pairs of the multigrid solver (see solver.cu learned_generate)
// ------------------------------------------------------------------------------------------
struct Mode {
    float kx, ky, kz, phase, amp;
};

// e[d][node] = sum over the modes of component d of amp cos(2 pi k.x + phase), 0 on fixed dofs
__global__ void k_random_field(int64_t nnx, int64_t nny, int64_t nn, float hx, float hy, float hz,
                               const Mode* __restrict__ modes, int per_comp, const uint8_t* __restrict__ fixed,
                               double* __restrict__ e) {
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const float x = (float)(node % nnx) * hx, y = (float)((node / nnx) % nny) * hy, z = (float)(node / (nnx * nny)) * hz;
    for (int d = 0; d < 3; ++d) {
        float s = 0.0f;
        for (int m = 0; m < per_comp; ++m) {
            const Mode md = modes[d * per_comp + m];
            s += md.amp * cospif(2.0f * (md.kx * x + md.ky * y + md.kz * z) + md.phase);
        }
        e[(int64_t)d * nn + node] = (fixed && fixed[node * 3 + d]) ? 0.0 : (double)s;
    }
}

void random_field(Context& c, Net& n, uint64_t seed, double* e) {
    const MeshDesc& m = c.mesh;
    const int per = 16;
    uint64_t s = seed * 0x2545F4914F6CDD1Dull + 17;
    auto unif = [&]() { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); };
    // the largest wavenumber of this sample: from 1 (smooth) up to half the mesh resolution
    const int kcap = std::max(1, std::min(m.nel[0], std::min(m.nel[1], m.nel[2])) / 2);
    const double kmax = 1.0 + unif() * (kcap - 1);
    std::vector<Mode> h((size_t)3 * per);
    for (auto& md : h) {
        md.kx = (float)std::floor(unif() * (kmax + 1.0));
        md.ky = (float)std::floor(unif() * (kmax + 1.0));
        md.kz = (float)std::floor(unif() * (kmax + 1.0));
        const double kk = std::sqrt((double)md.kx * md.kx + (double)md.ky * md.ky + (double)md.kz * md.kz);
        md.phase = (float)(2.0 * unif());
        md.amp = (float)((2.0 * unif() - 1.0) / (1.0 + kk));
    }
    n.modes.ensure(h.size() * sizeof(Mode));
    UWG_CUDA(cudaMemcpyAsync(n.modes.p, h.data(), h.size() * sizeof(Mode), cudaMemcpyHostToDevice, c.stream));
    LaunchScope ls(c, -1);
    k_random_field<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, 1.0f / m.nel[0], 1.0f / m.nel[1],
                                                          1.0f / m.nel[2], reinterpret_cast<const Mode*>(n.modes.p), per,
                                                          c.levels[0].fixed.p, e);
    UWG_CUDA(cudaStreamSynchronize(c.stream));   // the host mode table is released on return
}

// sample k: xs = (r / rms(r), v / rms(v)) (FP32, [6][nn]), ys = (e - v) / rms(v) ([3][nn])
__global__ void k_store_sample(int64_t n3, const double* __restrict__ r, const double* __restrict__ e,
                               const double* __restrict__ v, const double* __restrict__ sumsq, int64_t nvec,
                               float* __restrict__ xs, float* __restrict__ ys) {
    __shared__ double inv[2];
    if (threadIdx.x < 2)
        inv[threadIdx.x] = sumsq[threadIdx.x] > 0.0 ? 1.0 / sqrt(sumsq[threadIdx.x] / (double)nvec) : 0.0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n3) return;
    xs[i] = (float)(r[i] * inv[0]);
    xs[n3 + i] = (float)(v[i] * inv[1]);
    ys[i] = (float)((e[i] - v[i]) * inv[1]);
}

void dataset_reserve(Context& c, Net& n, int nsamples) {
    n.data_x.ensure((size_t)nsamples * 6 * n.nn);
    n.data_y.ensure((size_t)nsamples * 3 * n.nn);
    n.ysq.assign((size_t)nsamples, 0.0);
    n.nsamples = 0;
    prepare_viscosity(c, n);
}

void dataset_add(Context& c, Net& n, const double* r, const double* e, const double* v) {
    const int k = n.nsamples;
    UWG_REQUIRE((size_t)k < n.ysq.size(), UWGPU_ERR_ARGUMENT, "training set is full");
    n.sumsq.ensure(2);
    UWG_CUDA(cudaMemsetAsync(n.sumsq.p, 0, 2 * sizeof(double), c.stream));
    const int64_t n3 = 3 * n.nn;
    {
        LaunchScope ls(c, -1);
        k_sumsq<double><<<1, 1024, 0, c.stream>>>(n3, r, n.sumsq.p);
        k_sumsq<double><<<1, 1024, 0, c.stream>>>(n3, v, n.sumsq.p + 1);
    }
    float* xs = n.data_x.p + (size_t)k * 2 * n3;
    float* ys = n.data_y.p + (size_t)k * n3;
    {
        LaunchScope ls(c, -1);
        k_store_sample<<<nblk(n3, 256), 256, 0, c.stream>>>(n3, r, e, v, n.sumsq.p, n3, xs, ys);
    }
    UWG_CUDA(cudaMemsetAsync(n.sumsq.p, 0, sizeof(double), c.stream));
    {
        LaunchScope ls(c, -1);
        k_sumsq<float><<<1, 1024, 0, c.stream>>>(n3, ys, n.sumsq.p);
    }
    double h = 0.0;
    UWG_CUDA(cudaMemcpyAsync(&h, n.sumsq.p, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    n.ysq[(size_t)k] = h;
    n.nsamples = k + 1;
}

__global__ void k_scale_f(int64_t n, float a, float* __restrict__ x) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] *= a;
}

// the network's targets are scaled to unit RMS; out_scale maps its output back
void dataset_finish(Context& c, Net& n) {
    UWG_REQUIRE(n.nsamples > 0, UWGPU_ERR_STATE, "empty training set");
    double tot = 0.0;
    for (int k = 0; k < n.nsamples; ++k) tot += n.ysq[(size_t)k];
    const double rms = std::sqrt(tot / ((double)n.nsamples * 3.0 * n.nn));
    UWG_REQUIRE(rms > 0.0 && std::isfinite(rms), UWGPU_ERR_NAN, "training targets are zero or not finite");
    n.out_scale = (float)rms;
    const int64_t tot_n = (int64_t)n.nsamples * 3 * n.nn;
    LaunchScope ls(c, -1);
    k_scale_f<<<nblk(tot_n, 256), 256, 0, c.stream>>>(tot_n, (float)(1.0 / rms), n.data_y.p);
    for (auto& v : n.ysq) v /= rms * rms;
    UWG_CUDA(cudaStreamSynchronize(c.stream));
}

// ------------------------------------------------------------------------------------------
// Training: relative squared error per sample, Adam
// ------------------------------------------------------------------------------------------
__global__ void k_sample_input(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ xs,
                               const float* __restrict__ logeta, bf16* __restrict__ x0) {
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nn) return;
    const int64_t v = node_voxel(node, nnx, nny, g);
#pragma unroll
    for (int d = 0; d < 6; ++d) x0[v * kInChannels + d] = __float2bfloat16_rn(xs[(int64_t)d * nn + node]);
    x0[v * kInChannels + 6] = __float2bfloat16_rn(logeta[node]);
}

// loss += |out - y|^2 / ysq over free dofs; gout = 2 (out - y) / ysq there (0 elsewhere)
__global__ void k_rel_mse(int64_t nnx, int64_t nny, int64_t nn, Vol g, const float* __restrict__ out,
                          const float* __restrict__ y, const uint8_t* __restrict__ fixed, float inv_ysq,
                          float* __restrict__ gout, double* __restrict__ loss) {
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (node < nn) {
        const int64_t v = node_voxel(node, nnx, nny, g);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float diff = out[(int64_t)d * g.nv + v] - y[(int64_t)d * nn + node];
            if (fixed && fixed[node * 3 + d]) diff = 0.0f;
            gout[(int64_t)d * g.nv + v] = 2.0f * diff * inv_ysq;
            l = fmaf(diff * diff, inv_ysq, l);
        }
    }
    l = warp_sum(l);
    if ((threadIdx.x & 31) == 0 && loss) atomicAdd(loss, (double)l);
}

// one sample: forward, loss and its gradient, backward (grads accumulate); returns the loss
static void sample_step(Context& c, Net& n, int k, bool train, double* dloss) {
    const int64_t n3 = 3 * n.nn;
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        k_sample_input<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], n.data_x.p + (size_t)k * 2 * n3,
                                                               n.logeta.p, n.x0.p);
    }
    forward(c, n);
    UWG_CUDA(cudaMemsetAsync(n.gout.p, 0, (size_t)n.vol[0].nv * 3 * sizeof(float), c.stream));
    {
        LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
        const double ysq = n.ysq[(size_t)k];
        k_rel_mse<<<nblk(n.nn, 256), 256, 0, c.stream>>>(n.nnx, n.nny, n.nn, n.vol[0], n.out.p, n.data_y.p + (size_t)k * n3,
                                                          c.levels[0].fixed.p, ysq > 0.0 ? (float)(1.0 / ysq) : 0.0f,
                                                          n.gout.p, dloss);
    }
    if (train) backward(c, n);
}

void train(Context& c, Net& n, int epochs, int batch, float lr, uint64_t seed, double* train_loss,
           double* holdout_ratio) {
    UWG_REQUIRE(n.nsamples >= 2, UWGPU_ERR_STATE, "training needs at least two samples (learned_generate)");
    UWG_REQUIRE(epochs >= 0 && batch >= 1, UWGPU_ERR_ARGUMENT, "bad epochs or batch");
    const int nhold = std::max(1, n.nsamples / 10);
    const int ntrain = n.nsamples - nhold;
    std::vector<int> order((size_t)ntrain);
    for (int k = 0; k < ntrain; ++k) order[(size_t)k] = k;
    uint64_t s = seed ^ 0xA0761D6478BD642Full;
    DArray<double> dl;
    dl.ensure(2);
    double last = 0.0;
    for (int ep = 0; ep < epochs; ++ep) {
        for (int k = ntrain - 1; k > 0; --k) std::swap(order[(size_t)k], order[(size_t)(splitmix(s) % (uint64_t)(k + 1))]);
        UWG_CUDA(cudaMemsetAsync(dl.p, 0, sizeof(double), c.stream));
        for (int b0 = 0; b0 < ntrain; b0 += batch) {
            const int nb = std::min(batch, ntrain - b0);
            UWG_CUDA(cudaMemsetAsync(n.grads.p, 0, (size_t)n.nparams * sizeof(float), c.stream));
            for (int q = 0; q < nb; ++q) sample_step(c, n, order[(size_t)(b0 + q)], true, dl.p);
            n.adam_t++;
            const float b1 = 0.9f, b2 = 0.999f;
            const float bc1 = 1.0f - std::pow(b1, (float)n.adam_t), bc2 = 1.0f - std::pow(b2, (float)n.adam_t);
            {
                LaunchScope ls(c, UWGPU_KERNEL_LEARNED);
                k_adam<<<nblk(n.nparams, 256), 256, 0, c.stream>>>(n.nparams, n.params.p, n.grads.p, n.adam_m.p,
                                                                   n.adam_v.p, lr, b1, b2, 1e-8f, bc1, bc2, 1.0f / nb);
            }
            pack(c, n);
        }
        UWG_CUDA(cudaMemcpyAsync(c.host_scalars, dl.p, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
        UWG_CUDA(cudaStreamSynchronize(c.stream));
        last = c.host_scalars[0] / ntrain;
        if (!std::isfinite(last)) throw Error(UWGPU_ERR_NAN, "U-Net training diverged");
    }
    if (train_loss) *train_loss = last;
    // held-out samples: |y - N(x)|^2 / |y|^2 averaged (1 = no better than no correction)
    UWG_CUDA(cudaMemsetAsync(dl.p, 0, sizeof(double), c.stream));
    for (int k = ntrain; k < n.nsamples; ++k) sample_step(c, n, k, false, dl.p);
    UWG_CUDA(cudaMemcpyAsync(c.host_scalars, dl.p, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    UWG_CUDA(cudaStreamSynchronize(c.stream));
    if (holdout_ratio) *holdout_ratio = c.host_scalars[0] / nhold;
    check_errors(c, n);
}

}  // namespace unet
}  // namespace uwg
