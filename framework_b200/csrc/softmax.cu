// Softmax over one dimension and its backward: the step between S = Q.K^T and S.V in the
// attention-shaped use of the batched GEMM (ops/norm.rs:52-89, :125-163; kernels/softmax.cu).
// HBM-bound: the forward reads x once and writes out once (8 bytes per element), the backward reads
// dy and out once and writes dx once (12 bytes per element).  A row that fits a warp's registers
// (<= 2048 elements; <= 1024 where rows are not 16-byte aligned, as with an odd length) never leaves them between
// the max, the sum and the division; other shapes take a block-per-row or a block-per-32-columns loop over the same arithmetic.
#include "internal.h"

#include <algorithm>

namespace mni {

namespace {

constexpr int kRowsPerBlock = 8;   // one warp per row
constexpr float kNegInf = -__builtin_huge_valf();

__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Row in registers: lane l holds units l, l+32, ... (CH of them; unit index < len is live).  A unit is a float4 where the
// rows are 16-byte aligned, a float where they are not (an odd length): the warp's loads are contiguous either way.
__device__ __forceinline__ float unit_max(const float &v) { return v; }
__device__ __forceinline__ float unit_max(const float4 &v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }
__device__ __forceinline__ float unit_exp(float &v, float mx) { v = expf(v - mx); return v; }
__device__ __forceinline__ float unit_exp(float4 &v, float mx) {
    v.x = expf(v.x - mx); v.y = expf(v.y - mx);
    v.z = expf(v.z - mx); v.w = expf(v.w - mx);
    return (v.x + v.y) + (v.z + v.w);
}
__device__ __forceinline__ float unit_div(const float &v, float s) { return v / s; }
__device__ __forceinline__ float4 unit_div(const float4 &v, float s) { return make_float4(v.x / s, v.y / s, v.z / s, v.w / s); }
__device__ __forceinline__ float unit_dot(const float &g, const float &s) { return g * s; }
__device__ __forceinline__ float unit_dot(const float4 &g, const float4 &s) { return (g.x * s.x + g.y * s.y) + (g.z * s.z + g.w * s.w); }
__device__ __forceinline__ float unit_grad(const float &g, const float &s, float dot) { return s * (g - dot); }
__device__ __forceinline__ float4 unit_grad(const float4 &g, const float4 &s, float dot) {
    return make_float4(s.x * (g.x - dot), s.y * (g.y - dot), s.z * (g.z - dot), s.w * (g.w - dot));
}

// The row of this warp.  From the last one down: what the kernel before wrote last is what L2 still holds (scores of 100 MB
// between their product, this pass and the next product: attention 288 -> 277 us a pass, the forward's share 7, the backward's 5).
__device__ __forceinline__ long long last_rows_first() {
    return (gridDim.x - 1 - blockIdx.x) * static_cast<long long>(kRowsPerBlock) + (threadIdx.x >> 5);
}

template <typename V, int CH>
__global__ void __launch_bounds__(kRowsPerBlock * 32)
softmax_rows_fwd_kernel(const V *__restrict__ x, V *__restrict__ out, long long rows, int len) {
    grid_dependency_trigger();
    const long long row = last_rows_first();
    const int lane = threadIdx.x & 31;
    grid_dependency_wait();
    if (row >= rows) return;
    const V *xr = x + row * len;
    V v[CH];
    float mx = kNegInf;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int i = c * 32 + lane;
        if (i < len) {
            v[c] = __ldcs(xr + i);
            mx = fmaxf(mx, unit_max(v[c]));
        }
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c)
        if (c * 32 + lane < len) sum += unit_exp(v[c], mx);
    sum = warp_sum(sum);
    V *orow = out + row * len;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int i = c * 32 + lane;
        if (i < len) orow[i] = unit_div(v[c], sum);
    }
}

template <typename V, int CH>
__global__ void __launch_bounds__(kRowsPerBlock * 32)
softmax_rows_bwd_kernel(const V *__restrict__ dy, const V *__restrict__ out, V *__restrict__ dx, long long rows, int len) {
    grid_dependency_trigger();
    const long long row = last_rows_first();
    const int lane = threadIdx.x & 31;
    grid_dependency_wait();
    if (row >= rows) return;
    const V *gr = dy + row * len, *sr = out + row * len;
    V g[CH], s[CH];
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int i = c * 32 + lane;
        if (i < len) {
            g[c] = __ldcs(gr + i);
            s[c] = __ldcs(sr + i);
            dot += unit_dot(g[c], s[c]);
        }
    }
    dot = warp_sum(dot);
    V *drow = dx + row * len;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int i = c * 32 + lane;
        if (i < len) drow[i] = unit_grad(g[c], s[c], dot);
    }
}

// Any length, any alignment, inner == 1: one block per row, three passes over the row (the second
// and third hit L2 or L1).  Block reductions in a fixed order.
constexpr int kBlockThreads = 256;
__device__ __forceinline__ float block_reduce(float x, bool is_max) {
    __shared__ float ws[kBlockThreads / 32];
    __shared__ float result;
    x = is_max ? warp_max(x) : warp_sum(x);
    __syncthreads();                                 // ws / result may still be read from the last call
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = ws[0];
        for (int w = 1; w < kBlockThreads / 32; ++w) t = is_max ? fmaxf(t, ws[w]) : t + ws[w];
        result = t;
    }
    __syncthreads();
    return result;
}
__global__ void __launch_bounds__(kBlockThreads)
softmax_long_fwd_kernel(const float *__restrict__ x, float *__restrict__ out, long long len) {
    const float *xr = x + blockIdx.x * len;
    float *orow = out + blockIdx.x * len;
    float mx = kNegInf;
    for (long long i = threadIdx.x; i < len; i += kBlockThreads) mx = fmaxf(mx, xr[i]);
    mx = block_reduce(mx, true);
    float sum = 0.f;
    for (long long i = threadIdx.x; i < len; i += kBlockThreads) {
        const float e = expf(xr[i] - mx);
        orow[i] = e;
        sum += e;
    }
    sum = block_reduce(sum, false);
    for (long long i = threadIdx.x; i < len; i += kBlockThreads) orow[i] /= sum;
}
__global__ void __launch_bounds__(kBlockThreads)
softmax_long_bwd_kernel(const float *__restrict__ dy, const float *__restrict__ out, float *__restrict__ dx,
                        long long len) {
    const float *gr = dy + blockIdx.x * len, *sr = out + blockIdx.x * len;
    float *drow = dx + blockIdx.x * len;
    float dot = 0.f;
    for (long long i = threadIdx.x; i < len; i += kBlockThreads) dot += gr[i] * sr[i];
    dot = block_reduce(dot, false);
    for (long long i = threadIdx.x; i < len; i += kBlockThreads) drow[i] = sr[i] * (gr[i] - dot);
}

// inner > 1 (softmax over a dimension that is not the last): a block owns 32 neighbouring (outer, inner)
// columns, so every access is a coalesced 128-byte line, and its 8 warps split the dimension; the
// per-column max and sums meet in shared memory in warp order.
constexpr int kColWarps = 8;
__device__ __forceinline__ float cols_reduce(float x, bool is_max, float (*sh)[32]) {
    const int cx = threadIdx.x & 31, sg = threadIdx.x >> 5;
    __syncthreads();                                  // sh may still be read from the previous reduce
    sh[sg][cx] = x;
    __syncthreads();
    float t = sh[0][cx];
#pragma unroll
    for (int w = 1; w < kColWarps; ++w) t = is_max ? fmaxf(t, sh[w][cx]) : t + sh[w][cx];
    return t;
}
__global__ void __launch_bounds__(32 * kColWarps)
softmax_cols_fwd_kernel(const float *__restrict__ x, float *__restrict__ out, long long columns, long long dim,
                        long long inner) {
    __shared__ float sh[kColWarps][32];
    const int cx = threadIdx.x & 31, sg = threadIdx.x >> 5;
    const long long c = blockIdx.x * 32LL + cx;
    const bool live = c < columns;
    const long long base = live ? (c / inner) * dim * inner + (c % inner) : 0;
    float mx = kNegInf;
    if (live)
        for (long long s = sg; s < dim; s += kColWarps) mx = fmaxf(mx, x[base + s * inner]);
    mx = cols_reduce(mx, true, sh);
    float sum = 0.f;
    if (live)
        for (long long s = sg; s < dim; s += kColWarps) {
            const float e = expf(x[base + s * inner] - mx);
            out[base + s * inner] = e;
            sum += e;
        }
    sum = cols_reduce(sum, false, sh);
    if (live)
        for (long long s = sg; s < dim; s += kColWarps) out[base + s * inner] /= sum;   // own writes only
}
__global__ void __launch_bounds__(32 * kColWarps)
softmax_cols_bwd_kernel(const float *__restrict__ dy, const float *__restrict__ out, float *__restrict__ dx,
                        long long columns, long long dim, long long inner) {
    __shared__ float sh[kColWarps][32];
    const int cx = threadIdx.x & 31, sg = threadIdx.x >> 5;
    const long long c = blockIdx.x * 32LL + cx;
    const bool live = c < columns;
    const long long base = live ? (c / inner) * dim * inner + (c % inner) : 0;
    float dot = 0.f;
    if (live)
        for (long long s = sg; s < dim; s += kColWarps) dot += dy[base + s * inner] * out[base + s * inner];
    dot = cols_reduce(dot, false, sh);
    if (live)
        for (long long s = sg; s < dim; s += kColWarps)
            dx[base + s * inner] = out[base + s * inner] * (dy[base + s * inner] - dot);
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Units per lane of a row of `units`, rounded up to a compiled variant (0: the row does not fit `most` of them).
int chunks_for(long long units, int most) {
    const long long need = (units + 31) / 32;
    for (int ch : {1, 2, 4, 8, 16, 32})
        if (need <= ch) return ch <= most ? ch : 0;
    return 0;
}

template <typename V>
using RowsFwd = void (*)(const V *, V *, long long, int);
template <typename V>
using RowsBwd = void (*)(const V *, const V *, V *, long long, int);
template <typename V>
RowsFwd<V> rows_fwd(int ch) {
    switch (ch) {
        case 1: return softmax_rows_fwd_kernel<V, 1>;
        case 2: return softmax_rows_fwd_kernel<V, 2>;
        case 4: return softmax_rows_fwd_kernel<V, 4>;
        case 8: return softmax_rows_fwd_kernel<V, 8>;
        case 16: return softmax_rows_fwd_kernel<V, 16>;
        default: return softmax_rows_fwd_kernel<V, sizeof(V) == 4 ? 32 : 16>;
    }
}
template <typename V>
RowsBwd<V> rows_bwd(int ch) {
    switch (ch) {
        case 1: return softmax_rows_bwd_kernel<V, 1>;
        case 2: return softmax_rows_bwd_kernel<V, 2>;
        case 4: return softmax_rows_bwd_kernel<V, 4>;
        case 8: return softmax_rows_bwd_kernel<V, 8>;
        case 16: return softmax_rows_bwd_kernel<V, sizeof(V) == 4 ? 16 : 8>;
        default: return softmax_rows_bwd_kernel<V, sizeof(V) == 4 ? 32 : 8>;
    }
}

template <typename V>
int launch_rows_fwd(const float *x, float *out, int64_t rows, int64_t dim, int ch, cudaStream_t stream) {
    const dim3 grid(static_cast<unsigned>((rows + kRowsPerBlock - 1) / kRowsPerBlock));
    const cudaError_t e = launch_dependent(rows_fwd<V>(ch), grid, dim3(kRowsPerBlock * 32), 0, stream, reinterpret_cast<const V *>(x),
                                           reinterpret_cast<V *>(out), rows, static_cast<int>(dim * sizeof(float) / sizeof(V)));
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "softmax launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("softmax_rows_fwd");
    return MNI_B200_OK;
}
template <typename V>
int launch_rows_bwd(const float *dy, const float *out, float *dx, int64_t rows, int64_t dim, int ch, cudaStream_t stream) {
    const dim3 grid(static_cast<unsigned>((rows + kRowsPerBlock - 1) / kRowsPerBlock));
    const cudaError_t e = launch_dependent(rows_bwd<V>(ch), grid, dim3(kRowsPerBlock * 32), 0, stream, reinterpret_cast<const V *>(dy),
                                           reinterpret_cast<const V *>(out), reinterpret_cast<V *>(dx), rows,
                                           static_cast<int>(dim * sizeof(float) / sizeof(V)));
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "softmax launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("softmax_rows_bwd");
    return MNI_B200_OK;
}

}  // namespace

int launch_softmax_fwd(const float *x, float *out, int64_t outer, int64_t dim, int64_t inner, cudaStream_t stream) {
    if (outer * dim * inner == 0) return MNI_B200_OK;
    if (inner == 1) {
        // a lane holds up to 16 16-byte units (2048 elements a row), or up to 32 elements (1024) of a row that is not aligned
        const bool aligned = dim % 4 == 0 && aligned16(x) && aligned16(out);
        if (const int ch = aligned ? chunks_for(dim / 4, 16) : 0) return launch_rows_fwd<float4>(x, out, outer, dim, ch, stream);
        if (const int ch = aligned ? 0 : chunks_for(dim, 32)) return launch_rows_fwd<float>(x, out, outer, dim, ch, stream);
        softmax_long_fwd_kernel<<<static_cast<unsigned>(outer), kBlockThreads, 0, stream>>>(x, out, dim);
        MNI_LAUNCH_CHECK("softmax_long_fwd");
        return MNI_B200_OK;
    }
    const long long columns = outer * inner;
    softmax_cols_fwd_kernel<<<static_cast<unsigned>((columns + 31) / 32), 32 * kColWarps, 0, stream>>>(x, out, columns,
                                                                                                  dim, inner);
    MNI_LAUNCH_CHECK("softmax_cols_fwd");
    return MNI_B200_OK;
}

int launch_softmax_bwd(const float *dy, const float *out, float *dx, int64_t outer, int64_t dim, int64_t inner,
                       cudaStream_t stream) {
    if (outer * dim * inner == 0) return MNI_B200_OK;
    if (inner == 1) {
        const bool aligned = dim % 4 == 0 && aligned16(dy) && aligned16(out) && aligned16(dx);
        // two rows live in registers here: 1024 elements at most
        if (const int ch = aligned ? chunks_for(dim / 4, 8) : 0) return launch_rows_bwd<float4>(dy, out, dx, outer, dim, ch, stream);
        if (const int ch = aligned ? 0 : chunks_for(dim, 32)) return launch_rows_bwd<float>(dy, out, dx, outer, dim, ch, stream);
        softmax_long_bwd_kernel<<<static_cast<unsigned>(outer), kBlockThreads, 0, stream>>>(dy, out, dx, dim);
        MNI_LAUNCH_CHECK("softmax_long_bwd");
        return MNI_B200_OK;
    }
    const long long columns = outer * inner;
    softmax_cols_bwd_kernel<<<static_cast<unsigned>((columns + 31) / 32), 32 * kColWarps, 0, stream>>>(dy, out, dx,
                                                                                                  columns, dim, inner);
    MNI_LAUNCH_CHECK("softmax_cols_bwd");
    return MNI_B200_OK;
}

}  // namespace mni
