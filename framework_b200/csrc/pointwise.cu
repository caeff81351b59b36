// HBM-bound helpers around the GEMM: bias add, column sums (dbias), bias + GELU, device-side unbroadcast.
#include "activation.h"
#include "internal.h"

#include <algorithm>
#include <type_traits>

namespace mni {

namespace {

constexpr int kMaxDims = MNI_B200_MAX_DIMS;

int grid_for(long long work_items, int threads) {
    const long long blocks = (work_items + threads - 1) / threads;
    return static_cast<int>(std::max<long long>(1, std::min<long long>(blocks, device_sm_count() * 16LL)));
}

// ---- column sums -----------------------------------------------------------------------------------
// Block (bx, by) sums rows [by * rows_per, ...) of a 128-column strip (32 lanes x float4); its 8 warps take interleaved
// rows and are combined through shared memory in warp order.  The block that takes a strip's last ticket then adds
// the strip's slabs, warps again interleaved and combined in order, so the result does not depend on scheduling and
// one launch does what took two (and, with a copy of dy wanted, three): 5.5 -> 2.0 us of launches for a small layer.
// A strip summed by one block needs neither scratch nor ticket.
constexpr int kMaxStrips = 1024;             // several slabs per strip only up to this many strips (see colsum_slabs)
// Zero between launches.  Bank 1 belongs to the entry point that allocates nothing, whose partial sums are its own too: its
// calls may run beside the others'.
constexpr int kTicketBanks = 2;
__device__ unsigned int g_colsum_tickets[kTicketBanks * kMaxStrips];

__device__ __forceinline__ void store_cols(float *dst, long long col, long long n, const float4 &s) {
    dst[0] = s.x;
    if (col + 1 < n) dst[1] = s.y;
    if (col + 2 < n) dst[2] = s.z;
    if (col + 3 < n) dst[3] = s.w;
}
// Adds the 8 warps' values in warp order; the result is valid in warp 0.  AGAIN: red may still be read from an earlier fold.
template <bool AGAIN>
__device__ __forceinline__ float4 fold_warps(float4 (*red)[32], const float4 &acc) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (AGAIN) __syncthreads();
    red[warp][lane] = acc;
    __syncthreads();
    float4 s = red[0][lane];
    if (warp == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            s.x += red[w][lane].x; s.y += red[w][lane].y; s.z += red[w][lane].z; s.w += red[w][lane].w;
        }
    }
    return s;
}
// The end of a column-sum block: `acc` is this thread's sum over the block's rows.
__device__ __forceinline__ void finish_colsum(const float4 &acc, float4 (*red)[32], float *partial, float *out,
                                              long long n, int accumulate, int bank) {
    __shared__ unsigned int s_last;
    unsigned int *const ticket = g_colsum_tickets + bank * kMaxStrips + blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long col = (static_cast<long long>(blockIdx.x) * 32 + lane) * 4;
    float4 s = fold_warps<false>(red, acc);
    const int slabs = static_cast<int>(gridDim.y);
    if (slabs > 1) {
        if (warp == 0) {
            if (col < n) store_cols(partial + static_cast<long long>(blockIdx.y) * n + col, col, n, s);
            __threadfence();
            __syncwarp();
            if (lane == 0) s_last = atomicAdd(ticket, 1u) == static_cast<unsigned>(slabs - 1);
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (col < n) {
#pragma unroll 4
            for (int i = warp; i < slabs; i += 8) {
                const float *p = partial + static_cast<long long>(i) * n + col;
                t.x += __ldcg(p);
                if (col + 1 < n) t.y += __ldcg(p + 1);
                if (col + 2 < n) t.z += __ldcg(p + 2);
                if (col + 3 < n) t.w += __ldcg(p + 3);
            }
        }
        s = fold_warps<true>(red, t);
        if (threadIdx.x == 0) *ticket = 0u;
    }
    if (warp == 0 && col < n) {
        if (accumulate) {
            s.x += out[col];
            if (col + 1 < n) s.y += out[col + 1];
            if (col + 2 < n) s.z += out[col + 2];
            if (col + 3 < n) s.w += out[col + 3];
        }
        store_cols(out + col, col, n, s);
    }
}

template <bool COPY>
__global__ void __launch_bounds__(256)
colsum_kernel(const float *__restrict__ dy, long long ld, float *__restrict__ copy, float *__restrict__ partial,
              float *__restrict__ out, long long rows, long long n, long long rows_per, int accumulate, int bank) {
    __shared__ float4 red[8][32];
    grid_dependency_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long col = (static_cast<long long>(blockIdx.x) * 32 + lane) * 4;
    const long long r0 = blockIdx.y * rows_per;
    const long long r1 = min(rows, r0 + rows_per);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool vec = ((ld & 3) == 0) && ((reinterpret_cast<uintptr_t>(dy) & 15) == 0) && col + 3 < n &&
                     (!COPY || ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(copy) & 15) == 0));
    grid_dependency_wait();
    if (col < n) {
        long long r = r0 + warp;
        if (vec) {
            // eight rows in flight per thread, added in the same ascending order as the one-row loop
            constexpr int U = 8;
            for (; r + 8 * (U - 1) < r1; r += 8 * U) {
                float4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = __ldcs(reinterpret_cast<const float4 *>(dy + (r + 8 * u) * ld + col));
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (COPY) *reinterpret_cast<float4 *>(copy + (r + 8 * u) * n + col) = v[u];
                    acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w;
                }
            }
        }
#pragma unroll 4
        for (; r < r1; r += 8) {
            const float *p = dy + r * ld + col;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (vec) {
                v = __ldcs(reinterpret_cast<const float4 *>(p));
                if (COPY) *reinterpret_cast<float4 *>(copy + r * n + col) = v;
            } else {
                v.x = __ldcs(p);
                if (col + 1 < n) v.y = __ldcs(p + 1);
                if (col + 2 < n) v.z = __ldcs(p + 2);
                if (col + 3 < n) v.w = __ldcs(p + 3);
                if (COPY) store_cols(copy + r * n + col, col, n, v);
            }
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
    }
    finish_colsum(acc, red, partial, out, n, accumulate, bank);
}

// ---- bias + GELU (tanh form), the fused pointwise op that follows the MLP up-projection --------
// out[r, j] = f(y[r, j] + bias[j]), f the identity or GELU.  The tensor is one flat run, so four consecutive elements are
// a unit whatever n is; only the bias index wraps.  QUADS: the pointers allow 16-byte units (else an element each);
// ALIGNED: a unit's bias values are one aligned 16-byte load too.  `units` per launch stays below 2^31.
constexpr int kBiasUnits = 4;                // units in flight per thread
template <bool GELU>
__device__ __forceinline__ float bias_apply(float v) { return GELU ? gelu_tanh(v) : v; }
template <bool GELU, bool QUADS, bool ALIGNED>
__global__ void __launch_bounds__(256)
bias_kernel(const float *__restrict__ y, const float *__restrict__ bias, float *__restrict__ out, int units, int tail,
            FastDiv n) {
    grid_dependency_trigger();
    grid_dependency_wait();
    constexpr int W = QUADS ? 4 : 1;
    const int base = static_cast<int>(blockIdx.x) * (256 * kBiasUnits) + threadIdx.x;
    float v[kBiasUnits][W];
#pragma unroll
    for (int u = 0; u < kBiasUnits; ++u) {
        const int i = base + u * 256;
        if (i >= units) continue;
        if (QUADS) *reinterpret_cast<float4 *>(v[u]) = *reinterpret_cast<const float4 *>(y + 4ll * i);
        else v[u][0] = y[i];
    }
#pragma unroll
    for (int u = 0; u < kBiasUnits; ++u) {
        const int i = base + u * 256;
        if (i >= units) continue;
        if (ALIGNED) {                       // n counts units here
            const int c = i - fd_div(i, n) * static_cast<int>(n.d);
            const float4 b = __ldg(reinterpret_cast<const float4 *>(bias) + c);
            const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < W; ++e) v[u][e] = bias_apply<GELU>(v[u][e] + bb[e]);
        } else {
            const int at = i * W;
            int c = at - fd_div(at, n) * static_cast<int>(n.d);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                v[u][e] = bias_apply<GELU>(v[u][e] + __ldg(bias + c));
                if (++c == static_cast<int>(n.d)) c = 0;
            }
        }
        if (QUADS) *reinterpret_cast<float4 *>(out + 4ll * i) = *reinterpret_cast<float4 *>(v[u]);
        else out[i] = v[u][0];
    }
    // the last, partial unit
    if (QUADS && blockIdx.x == 0 && static_cast<int>(threadIdx.x) < tail) {
        const int at = units * 4 + static_cast<int>(threadIdx.x);
        const int c = at - fd_div(at, n) * static_cast<int>(n.d);
        out[at] = bias_apply<GELU>(y[at] + __ldg(bias + c));
    }
}

// Backward: dx = grad * gelu'(x + bias) written once, and the column sums of dx (same block shape and fixed summation
// order as colsum_kernel; no atomics on values).
__global__ void __launch_bounds__(256, 4)      // four blocks per SM is what colsum_slabs plans for: one wave
bias_gelu_bwd_kernel(const float *__restrict__ grad, const float *__restrict__ x, const float *__restrict__ bias,
                     float *__restrict__ dx, float *__restrict__ partial, float *__restrict__ dbias, long long rows,
                     long long n, long long rows_per, int accumulate) {
    __shared__ float4 red[8][32];
    grid_dependency_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long col = (static_cast<long long>(blockIdx.x) * 32 + lane) * 4;
    const long long r0 = blockIdx.y * rows_per;
    const long long r1 = min(rows, r0 + rows_per);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool vec = ((n & 3) == 0) && col + 3 < n &&
                     (((reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(x) |
                        reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(bias)) & 15) == 0);
    grid_dependency_wait();
    if (col < n) {
        float b[4] = {0.f, 0.f, 0.f, 0.f};
        for (int e = 0; e < 4; ++e)
            if (col + e < n) b[e] = __ldg(bias + col + e);
        long long r = r0 + warp;
        if (vec) {
            auto batch = [&](auto rows_in_flight) {
                constexpr int U = decltype(rows_in_flight)::value;
                for (; r + 8 * (U - 1) < r1; r += 8 * U) {
                    float4 g[U], v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        g[u] = __ldcs(reinterpret_cast<const float4 *>(grad + (r + 8 * u) * n + col));
                        v[u] = __ldcs(reinterpret_cast<const float4 *>(x + (r + 8 * u) * n + col));
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        float4 d;
                        d.x = g[u].x * gelu_tanh_grad(v[u].x + b[0]);
                        d.y = g[u].y * gelu_tanh_grad(v[u].y + b[1]);
                        d.z = g[u].z * gelu_tanh_grad(v[u].z + b[2]);
                        d.w = g[u].w * gelu_tanh_grad(v[u].w + b[3]);
                        *reinterpret_cast<float4 *>(dx + (r + 8 * u) * n + col) = d;
                        acc.x += d.x; acc.y += d.y; acc.z += d.z; acc.w += d.w;
                    }
                }
            };
            batch(std::integral_constant<int, 2>{});      // rows in flight per thread (four spill at 64 registers)
            batch(std::integral_constant<int, 1>{});
        } else {
            for (; r < r1; r += 8) {
                const long long off = r * n + col;
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                for (int e = 0; e < 4; ++e) {
                    if (col + e < n) {
                        d[e] = __ldg(grad + off + e) * gelu_tanh_grad(__ldg(x + off + e) + b[e]);
                        dx[off + e] = d[e];
                    }
                }
                acc.x += d[0]; acc.y += d[1]; acc.z += d[2]; acc.w += d[3];
            }
        }
    }
    finish_colsum(acc, red, partial, dbias, n, accumulate, 0);
}

struct UnbArgs {
    int nd;                      // dims of the original (small) shape, right-aligned into the grad shape
    long long oshape[kMaxDims];  // original shape
    long long gstride[kMaxDims]; // grad stride of the matching grad dim
    int nred;                    // number of reduced (broadcast) dims incl. leading extra dims
    long long rshape[kMaxDims];  // extents of reduced dims, outermost first
    long long rstride[kMaxDims]; // grad strides of reduced dims
    long long rtotal;
    long long total;
};
// One thread per element of the original shape; it sums the grad elements that
// broadcast onto it in ascending flat order -- the order utils::unbroadcast adds them.
__global__ void unbroadcast_kernel(const float *__restrict__ grad, float *__restrict__ out, const UnbArgs a,
                                   int accumulate) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < a.total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        long long rem = i, base = 0;
        for (int d = a.nd - 1; d >= 0; --d) {
            const long long q = rem % a.oshape[d];
            rem /= a.oshape[d];
            base += q * a.gstride[d];
        }
        float s = 0.f;
        for (long long r = 0; r < a.rtotal; ++r) {
            long long rr = r, off = base;
            for (int d = a.nred - 1; d >= 0; --d) {
                off += (rr % a.rshape[d]) * a.rstride[d];
                rr /= a.rshape[d];
            }
            s += grad[off];
        }
        out[i] = accumulate ? out[i] + s : s;
    }
}

}  // namespace

namespace {
template <bool GELU>
int launch_bias(const float *y, const float *bias, float *out, int64_t rows, int64_t n, cudaStream_t stream) {
    if (rows == 0 || n == 0) return MNI_B200_OK;
    // The kernel's flat index stays below 2^31, the last block's included: longer rows go out in pieces of columns.
    constexpr int64_t kMostUnits = (1LL << 31) - 8192, kPiece = 1LL << 30;
    if (n > kMostUnits) {
        for (int64_t r = 0; r < rows; ++r)
            for (int64_t c = 0; c < n; c += kPiece) {
                const int rc = launch_bias<GELU>(y + r * n + c, bias + c, out + r * n + c, 1, std::min(kPiece, n - c), stream);
                if (rc) return rc;
            }
        return MNI_B200_OK;
    }
    const bool quads = ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    const bool aligned = quads && n % 4 == 0 && (reinterpret_cast<uintptr_t>(bias) & 15) == 0;
    // whole groups of rows per launch, so that every launch's flat index stays below 2^31 and its start keeps the
    // alignment (a multiple of four rows)
    const int64_t limit = kMostUnits / n;
    const int64_t step = std::max<int64_t>(1, limit >= 4 ? limit / 4 * 4 : limit);
    for (int64_t r = 0; r < rows; r += step) {
        const int64_t total = std::min(step, rows - r) * n;
        const float *ys = y + r * n;
        float *os = out + r * n;
        const bool q = quads && (r * n) % 4 == 0;
        const int units = static_cast<int>(q ? total / 4 : total), tail = static_cast<int>(q ? total % 4 : 0);
        const dim3 grid(static_cast<unsigned>(std::max(1, (units + 256 * kBiasUnits - 1) / (256 * kBiasUnits))));
        const FastDiv fd = make_fastdiv(aligned && q ? n / 4 : n);
        const cudaError_t e = launch_dependent(aligned && q ? bias_kernel<GELU, true, true>
                                               : q          ? bias_kernel<GELU, true, false>
                                                            : bias_kernel<GELU, false, false>,
                                               grid, dim3(256), 0, stream, ys, bias, os, units, tail, fd);
        if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "bias_kernel launch failed: %s", cudaGetErrorString(e));
        MNI_LAUNCH_CHECK("bias_kernel");
    }
    return MNI_B200_OK;
}
}  // namespace

int launch_add_bias(const float *y, const float *bias, float *out, int64_t rows, int64_t n, cudaStream_t stream) {
    return launch_bias<false>(y, bias, out, rows, n, stream);
}
int launch_bias_gelu(const float *x, const float *bias, float *out, int64_t rows, int64_t n, cudaStream_t stream) {
    return launch_bias<true>(x, bias, out, rows, n, stream);
}

// Slabs of rows per 128-column strip: about four blocks per SM in all, every warp of a block at least eight rows.
static int colsum_slabs(int64_t rows, int64_t n, int sm_count) {
    const long long strips = (n + 127) / 128;
    if (strips > kMaxStrips) return 1;
    long long slabs = std::max<long long>(1, (sm_count * 4LL) / strips);
    slabs = std::min<long long>(slabs, (rows + 63) / 64);
    return static_cast<int>(std::max<long long>(1, slabs));
}

size_t colsum_partial_bytes(int64_t rows, int64_t n, int sm_count) {
    return static_cast<size_t>(colsum_slabs(rows, n, sm_count)) * n * sizeof(float);
}

int launch_colsum(const float *dy, int64_t ld, float *copy, float *out, int64_t rows, int64_t n, bool accumulate,
                  float *partial, int sm_count, cudaStream_t stream, int ticket_bank) {
    if (n == 0) return MNI_B200_OK;
    const int slabs = colsum_slabs(rows, n, sm_count);
    const long long rows_per = (rows + slabs - 1) / slabs;
    dim3 grid(static_cast<unsigned>((n + 127) / 128), static_cast<unsigned>(slabs));
    const cudaError_t e = launch_dependent(copy ? colsum_kernel<true> : colsum_kernel<false>, grid, dim3(256), 0, stream, dy,
                                           ld, copy, partial, out, rows, n, rows_per, accumulate ? 1 : 0, ticket_bank);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "colsum_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("colsum_kernel");
    return MNI_B200_OK;
}

int launch_bias_gelu_bwd(const float *grad, const float *x, const float *bias, float *dx, float *dbias,
                         int64_t rows, int64_t n, bool accumulate, float *partial, int sm_count,
                         cudaStream_t stream) {
    if (n == 0 || rows == 0) return MNI_B200_OK;
    const int slabs = colsum_slabs(rows, n, sm_count);
    const long long rows_per = (rows + slabs - 1) / slabs;
    dim3 grid(static_cast<unsigned>((n + 127) / 128), static_cast<unsigned>(slabs));
    const cudaError_t e = launch_dependent(bias_gelu_bwd_kernel, grid, dim3(256), 0, stream, grad, x, bias, dx, partial, dbias,
                                           rows, n, rows_per, accumulate ? 1 : 0);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "bias_gelu_bwd_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("bias_gelu_bwd_kernel");
    return MNI_B200_OK;
}

int launch_copy(const float *src, float *dst, int64_t n, cudaStream_t stream) {
    if (n == 0 || src == dst || dst == nullptr) return MNI_B200_OK;
    MNI_CUDA(cudaMemcpyAsync(dst, src, static_cast<size_t>(n) * sizeof(float), cudaMemcpyDeviceToDevice, stream));
    return MNI_B200_OK;
}

int launch_unbroadcast(const float *grad, const int64_t *gshape, int gnd, const int64_t *oshape, int ond,
                       float *out, bool accumulate, cudaStream_t stream) {
    long long gstr[kMaxDims];
    long long acc = 1;
    for (int d = gnd - 1; d >= 0; --d) { gstr[d] = acc; acc *= gshape[d]; }
    UnbArgs a{};
    a.nd = ond;
    a.total = 1;
    a.rtotal = 1;
    a.nred = 0;
    const int off = gnd - ond;
    for (int d = 0; d < off; ++d) {           // leading dims the original does not have
        a.rshape[a.nred] = gshape[d];
        a.rstride[a.nred] = gstr[d];
        a.rtotal *= gshape[d];
        ++a.nred;
    }
    for (int d = 0; d < ond; ++d) {
        a.oshape[d] = oshape[d];
        a.total *= oshape[d];
        if (oshape[d] == 1 && gshape[d + off] != 1) {
            a.gstride[d] = 0;
            a.rshape[a.nred] = gshape[d + off];
            a.rstride[a.nred] = gstr[d + off];
            a.rtotal *= gshape[d + off];
            ++a.nred;
        } else {
            a.gstride[d] = gstr[d + off];
        }
    }
    if (a.total == 0) return MNI_B200_OK;
    unbroadcast_kernel<<<grid_for(a.total, 256), 256, 0, stream>>>(grad, out, a, accumulate ? 1 : 0);
    MNI_LAUNCH_CHECK("unbroadcast_kernel");
    return MNI_B200_OK;
}

}  // namespace mni
