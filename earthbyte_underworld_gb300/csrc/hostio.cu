// Layout changes at the boundary to host memory.
//
// The device keeps vectors by component ([d][node], [d][slot]) and element data by entry ([k][element]);
// the host arrays of the C ABI are by node, slot and element.  The change of layout runs on the device, at
// memory bandwidth, on its way to or from a plain copy: done on the host (a scalar loop over a temporary) it
// took most of a call: 40 of 44 ms for the element matrices of a 32^3 mesh, 7 of 8.6 ms for the mapping of
// 2.4M points.  Staging memory is bounded: larger transfers, either way, go in pieces of kIoBytes.
#include <algorithm>

#include "internal.cuh"

namespace uwg {

namespace {

constexpr size_t kIoBytes = (size_t)64 << 20;

// the components of nodes first + i, i < count, of n
template <int DIM, typename T>
__global__ void k_from_nodes(int64_t n, int64_t first, int64_t count, const double* __restrict__ a, T* __restrict__ soa) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
#pragma unroll
    for (int d = 0; d < DIM; ++d) soa[(int64_t)d * n + first + i] = (T)a[i * DIM + d];
}

// out[i][0 .. W) of items first + i, i < count: the DIM components, then zeros
template <int DIM, int W, typename T>
__global__ void k_to_items(int64_t n, int64_t first, int64_t count, const T* __restrict__ soa, double* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;   // one value per thread: stores coalesce
    if (t >= count * W) return;
    const int64_t i = t / W;
    const int d = (int)(t - i * W);
    out[t] = d < DIM ? (double)soa[(int64_t)d * n + first + i] : 0.0;
}

// out[i][k] = src[k][first + i]: tiles of 32 x 32 through shared memory
__global__ void __launch_bounds__(256) k_entries_out(int entries, int64_t ne, int64_t first, int64_t count,
                                                     const double* __restrict__ src, double* __restrict__ out) {
    __shared__ double tile[32][33];
    const int64_t e0 = (int64_t)blockIdx.x * 32;
    const int k0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int k = ty; k < 32; k += 8)
        if (k0 + k < entries && e0 + tx < count) tile[k][tx] = src[(int64_t)(k0 + k) * ne + first + e0 + tx];
    __syncthreads();
    for (int e = ty; e < 32; e += 8)
        if (k0 + tx < entries && e0 + e < count) out[(e0 + e) * entries + k0 + tx] = tile[tx][e];
}

// Full symmetric element matrices from their packed upper triangles: a block stages 32 elements' entries
// ([k][32], rows padded: the reads along a matrix row then fall on different banks) and writes each
// matrix as one contiguous run.  Bound by the writes: 4.6 KB per 3D element.
template <int DIM>
__global__ void __launch_bounds__(256) k_unpack_ke(int64_t ne, int64_t first, int64_t count,
                                                   const double* __restrict__ Kp, double* __restrict__ out) {
    constexpr int ND = (1 << DIM) * DIM, NP = ND * (ND + 1) / 2;
    extern __shared__ double sk[];   // NP x 33
    const int64_t e0 = (int64_t)blockIdx.x * 32;
    const int here = (int)min((int64_t)32, count - e0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (tx < here)
        for (int k = ty; k < NP; k += 8) sk[k * 33 + tx] = Kp[(int64_t)k * ne + first + e0 + tx];
    __syncthreads();
    for (int t = threadIdx.x; t < here * ND * ND; t += 256) {
        const int e = t / (ND * ND), rc = t - e * (ND * ND), r = rc / ND, c = rc - r * ND;
        const int lo = min(r, c), hi = max(r, c);
        out[e0 * (ND * ND) + t] = sk[packed_index(ND, lo, hi) * 33 + e];
    }
}

// Runs make(first, count, staging) and a copy to `host` for pieces of the items, `width` values each
template <typename F>
void in_pieces(Context& c, int64_t items, int64_t width, double* host, F&& make) {
    const int64_t step = std::max<int64_t>(1, (int64_t)(kIoBytes / (sizeof(double) * (size_t)width)));
    c.io.ensure((size_t)(std::min(items, step) * width));
    for (int64_t first = 0; first < items; first += step) {
        const int64_t count = std::min(step, items - first);
        {
            LaunchScope ls(c, -1);
            make(first, count, c.io.p);
        }
        check_launch("layout change");
        UWG_CUDA(cudaMemcpyAsync(host + first * width, c.io.p, (size_t)(count * width) * sizeof(double),
                                 cudaMemcpyDeviceToHost, c.stream));
    }
}

}  // namespace

// soa[d][node] (device, T) = host[node][d]
template <typename T>
void vector_from_host(Context& c, int64_t n, int dim, const double* host, T* soa) {
    if (n == 0) return;
    const int64_t step = (int64_t)(kIoBytes / (sizeof(double) * (size_t)dim));
    c.io.ensure((size_t)(std::min(n, step) * dim));
    for (int64_t first = 0; first < n; first += step) {
        const int64_t count = std::min(step, n - first);
        UWG_CUDA(cudaMemcpyAsync(c.io.p, host + first * dim, (size_t)(count * dim) * sizeof(double), cudaMemcpyHostToDevice,
                                 c.stream));
        LaunchScope ls(c, -1);
        if (dim == 3) k_from_nodes<3, T><<<blocks_for(count, 256), 256, 0, c.stream>>>(n, first, count, c.io.p, soa);
        else k_from_nodes<2, T><<<blocks_for(count, 256), 256, 0, c.stream>>>(n, first, count, c.io.p, soa);
    }
    check_launch("k_from_nodes");
}

// host[item][0 .. width) = soa[d][item], zeros past the dimension (width: dim or 3)
template <typename T>
void vector_to_host(Context& c, int64_t n, int dim, int width, const T* soa, double* host) {
    if (n == 0) return;
    in_pieces(c, n, width, host, [&](int64_t first, int64_t count, double* out) {
        const unsigned b = blocks_for(count * width, 256);
        if (dim == 3) k_to_items<3, 3, T><<<b, 256, 0, c.stream>>>(n, first, count, soa, out);
        else if (width == 3) k_to_items<2, 3, T><<<b, 256, 0, c.stream>>>(n, first, count, soa, out);
        else k_to_items<2, 2, T><<<b, 256, 0, c.stream>>>(n, first, count, soa, out);
    });
}

// host[i][k] = src[k][first + i] of `count` elements of ne
void entries_to_host(Context& c, int entries, int64_t ne, int64_t first, int64_t count, const double* src, double* host) {
    in_pieces(c, count, entries, host, [&](int64_t f, int64_t n, double* out) {
        const dim3 grid(blocks_for(n, 32), (unsigned)((entries + 31) / 32));
        k_entries_out<<<grid, 256, 0, c.stream>>>(entries, ne, first + f, n, src, out);
    });
}

// host[i] = the full element matrix of element first + i, from the packed triangles Kp[k][e]
void element_matrices_to_host(Context& c, int64_t first, int64_t count, const double* Kp, double* host) {
    const int64_t ne = c.mesh.ne;
    const int nd = c.mesh.dim << c.mesh.dim;
    const size_t smem = (size_t)packed_size(nd) * 33 * sizeof(double);
    if (c.mesh.dim == 3)
        UWG_CUDA(cudaFuncSetAttribute(k_unpack_ke<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    in_pieces(c, count, (int64_t)nd * nd, host, [&](int64_t f, int64_t n, double* out) {
        if (c.mesh.dim == 3) k_unpack_ke<3><<<blocks_for(n, 32), 256, smem, c.stream>>>(ne, first + f, n, Kp, out);
        else k_unpack_ke<2><<<blocks_for(n, 32), 256, smem, c.stream>>>(ne, first + f, n, Kp, out);
    });
}

template void vector_from_host<double>(Context&, int64_t, int, const double*, double*);
template void vector_from_host<float>(Context&, int64_t, int, const double*, float*);
template void vector_to_host<double>(Context&, int64_t, int, int, const double*, double*);
template void vector_to_host<float>(Context&, int64_t, int, int, const float*, double*);

}  // namespace uwg
