// A few rows (at most 16) against a large weight, in the split TF32 arithmetic of the tensor path:
//
//   forward : y[M,N]  = x[M,K] . W[K,N] (+ bias)
//   dx      : dx[M,K] = dy[M,N] . W[K,N]^T
//
// Bound by HBM: the weight is read once, 67 MB = 10.3 us at K = N = 4096 of the measured copy rate.  The
// warp-level mma.sync is the right matrix instruction here although tcgen05 is several times faster per SM: the
// 805 M multiply-adds of 16 rows are 5 us of it spread over the warps that stream the weight, with no tensor memory to
// allocate, no descriptors, no operand staging beyond the ring and an accumulator that is already in registers.  The
// tcgen05 path takes the same products in 64-wide tiles with a split contraction and a second kernel that sums it, and
// gathers a weight with an odd row length into scratch first.  Nine rows x 4096 x 4096: forward 20.1 -> 18.0 us, dx 19.9 ->
// 18.0; 4096 x 4095: forward 53 -> 21 us, dx 44 -> 22.
//
// Split as in the tensor path: hi = x with the low 13 mantissa bits cut, lo = x - hi, products lo.hi + hi.lo + hi.hi.
// A chain in the tensor core's accumulator, which truncates, is kFlush elements long; longer sums are added up in
// registers, and the slices of the contraction in ascending order.
#include "device_utils.h"
#include "internal.h"

#include <algorithm>

namespace mni {

namespace {

constexpr int kWarps = 4;                    // each streams 32 x 32 tiles of the weight
constexpr int kThreads = 32 * kWarps;
constexpr int kDepth = 4;                    // 32 x 32 weight tiles held per warp, three in flight: 96 KB per SM with two blocks
constexpr int kRows = 16;
constexpr int kFlush = 256;                  // contraction elements summed in one tensor-core accumulator
// Contraction elements of x staged at a time, in two buffers where a block's slice is longer.  128-wide strips: 33 KB
// either way, which leaves room for two blocks per SM; 32-wide ones, whose warps take every fourth tile each, need chunks of
// four tiles per warp for the copies to be in time.
constexpr int kChunk = 256, kChunkNarrow = 512;
constexpr int64_t kMaxTotal = 16384;         // longest contraction taken here
constexpr int kMaxSlices = 8;                // slices of a strip: one portable cluster

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void split(float x, uint32_t &hi, uint32_t &lo) {
    hi = __float_as_uint(x) & 0xFFFFE000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
// acc += a . b in three passes, for the four 8-column tiles of a warp.
__device__ __forceinline__ void mma_split(float (&acc)[4][4], const uint32_t (&ah)[4], const uint32_t (&al)[4],
                                          const float (&b0)[4], const float (&b1)[4]) {
    uint32_t h0[4], l0[4], h1[4], l1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { split(b0[j], h0[j], l0[j]); split(b1[j], h1[j], l1[j]); }
    // pass by pass, so that neighbouring instructions work on different accumulators
#pragma unroll
    for (int j = 0; j < 4; ++j) mma_tf32(acc[j], al, h0[j], h1[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) mma_tf32(acc[j], ah, l0[j], l1[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) mma_tf32(acc[j], ah, h0[j], h1[j]);
}

// out[m, o] = sum_c x[m, c] . w(c, o), with w(c, o) = W[c, o] (forward) or W[o, c] (DX).
// grid = (strips of outputs, contraction slices), the slices of a strip one cluster.  WK = 1: the block's four warps take
// 32 outputs each of a 128-wide strip; WK = 4: they share a 32-wide strip and take every fourth tile of the slice each,
// which keeps more of the chip busy when the outputs are few.  Every warp streams its part of W through a private ring of
// 32 x 32 tiles by cp.async of 16-byte units; x is staged once per block in the same way.  Rows that are not 16-byte
// aligned (VEC = false) are copied from the boundary before them, nine units for 32 words, and keep their shift in shared
// memory, where the fragment reads add it.  (Copied word by word they took the load path 26 cycles per 128 bytes: 16 rows x
// 4096 x 4095 forward 30 -> 20.8 us, dx 34 -> 22; 3 rows x 5486 x 7657 127 -> 85.)  The tile pitch makes the fragment
// reads of aligned rows conflict-free: 40 floats for 16-byte reads of four neighbouring outputs (forward), 36 for reads
// down a column (DX).  The slices' sums meet through distributed shared memory.
template <bool DX, bool VEC, int WK>
__global__ void __launch_bounds__(kThreads, 2)
rows_kernel(const float *__restrict__ x, long long ldx, const float *__restrict__ W, long long ldw, float *__restrict__ y,
            long long ldy, const float *__restrict__ bias, int accumulate, int M, long long outs, long long total, int k_per,
            int y_vec) {
    constexpr int PITCH = DX ? 36 : 40;
    constexpr int OUTS = 32 * (kWarps / WK), SUM_PITCH = OUTS + 4;      // outputs per block
    extern __shared__ __align__(16) float smem[];
    constexpr int CHUNK = WK == 1 ? kChunk : kChunkNarrow;
    const int xk = k_per <= 512 ? k_per : CHUNK;            // contraction per chunk of x
    const int xp = xk + 4;                                  // = 4 mod 32: the A fragments' scalar reads hit all banks
    float *xs = smem;                                       // [1 or 2][kRows][xp]
    float *ring = smem + kRows * xp * (k_per <= 512 ? 1 : 2);   // [warps][depth][32][PITCH]; later the block's sums
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const long long k0 = static_cast<long long>(blockIdx.y) * k_per;
    const int kc = static_cast<int>(min(static_cast<long long>(k_per), total - k0));
    const int ow = warp / WK, kw = warp % WK;               // this warp's 32 outputs within the block, its share of the tiles
    const long long o0 = static_cast<long long>(blockIdx.x) * OUTS + ow * 32;
    const int nb = ((kc + 31) / 32 - kw + WK - 1) / WK;     // tiles kw, kw + WK, ... of the slice
    float *mine = ring + warp * (kDepth * 32 * PITCH);
    // extents of this warp's part of W, as rows and columns of W (tiles start at multiples of 32 of either)
    const int rows_live = DX ? static_cast<int>(max(0ll, min(32ll, outs - o0))) : kc;
    const int cols_live = DX ? kc : static_cast<int>(max(0ll, min(32ll, outs - o0)));
    const float *wp = DX ? W + o0 * ldw + k0 : W + k0 * ldw + o0;
    // Words by which a row starts past a 16-byte boundary; rows four apart are alike, so the row that a lane copies or
    // multiplies has one shift throughout.
    const int w_at = static_cast<int>((reinterpret_cast<uintptr_t>(wp) >> 2) & 3), w_step = static_cast<int>(ldw & 3);
    auto shift_of = [&](int row) { return VEC ? 0 : (w_at + row * w_step) & 3; };
    const int x_at = static_cast<int>((reinterpret_cast<uintptr_t>(x) >> 2) & 3), x_step = static_cast<int>(ldx & 3);
    auto x_shift = [&](int m) { return (x_at + m * x_step) & 3; };
    grid_dependency_trigger();
    grid_dependency_wait();
    auto issue = [&](int b) {
        if (b < nb) {
            float *slot = mine + (b % kDepth) * (32 * PITCH);
            const int at = (b * WK + kw) * 32, r0 = DX ? 0 : at, c0 = DX ? at : 0;
            if (VEC) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = i * 4 + (lane >> 3), c = (lane & 7) * 4;
                    const bool ok = r0 + r < rows_live && c0 + c < cols_live;
                    cp_async16(slot + r * PITCH + c, ok ? wp + (r0 + r) * ldw + c0 + c : W, ok);
                }
            } else {
                // whole 16-byte units from the boundary before the row's part: nine cover 32 words at any shift
                const int end = min(32, cols_live - c0);
                auto unit = [&](int r, int q, int sh) {
                    const int words = r0 + r < rows_live && end > 0 ? max(0, min(4, end + sh - 4 * q)) : 0;
                    const float *src = words > 0 ? wp + (r0 + r) * ldw + c0 - sh + 4 * q : x - x_at;
                    cp_async16_part(slot + r * PITCH + 4 * q, src, 4 * words);
                };
                const int sh = shift_of(lane >> 3), sh_last = shift_of(lane);
#pragma unroll
                for (int i = 0; i < 8; ++i) unit(i * 4 + (lane >> 3), lane & 7, sh);
                if (sh_last > 0) unit(lane, 8, sh_last);
            }
        }
        cp_async_commit();                                  // empty groups keep the count uniform
    };
    const int quads = xk / 4 + 1;
    auto stage_x = [&](int chunk) {
        const int at = chunk * xk, live = min(xk, kc - at);
        float *dst = xs + (chunk & 1) * (kRows * xp);
        for (int i = threadIdx.x; i < kRows * quads; i += kThreads) {
            const int m = i / quads, q = i - m * quads, sh = x_shift(m);
            const int words = m < M ? max(0, min(4, live + sh - 4 * q)) : 0;
            cp_async16_part(dst + m * xp + 4 * q, words > 0 ? x + m * ldx + k0 + at - sh + 4 * q : x - x_at, 4 * words);
        }
    };
    stage_x(0);
    cp_async_commit();
#pragma unroll
    for (int b = 0; b < kDepth - 1; ++b) issue(b);
    cp_async_wait<kDepth - 1>();                            // x (the oldest group) has landed
    __syncthreads();
    float acc[4][4], sum[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = sum[j][e] = 0.f;
    // the same for all warps; a slice of one chunk never comes to its end
    const int rounds = ((kc + 31) / 32 + WK - 1) / WK, chunk_tiles = k_per <= 512 ? rounds : CHUNK / (32 * WK);
    const float *xr = xs + g * xp + x_shift(g) + kw * 32 + t;
    int turn = 0, chunk = 0;                                // the tile with which the next chunk of x begins
    for (int b = 0; b < rounds; ++b, xr += 32 * WK) {
        __syncwarp();                                       // every lane is done with the slot that is filled next
        issue(b + kDepth - 1);
        cp_async_wait<kDepth - 1>();                        // tile b has landed, for this lane ...
        if (b == turn) {
            // This chunk of x, staged at least four groups ago, has landed for every thread, and every warp is done with the
            // chunk before: the next one takes its place, as part of the next tile's group.
            if (chunk > 0) {
                __syncthreads();
                xr += ((chunk & 1) ? kRows * xp : -kRows * xp) - xk;
            }
            turn += chunk_tiles;
            if (++chunk * xk < kc) stage_x(chunk);
        }
        __syncwarp();                                       // ... and for the others
        if (WK > 1 && b >= nb) continue;
        const float *slot = mine + (b % kDepth) * (32 * PITCH);
        const float *rows = slot + shift_of(DX ? g : t);    // of the row whose elements this lane multiplies
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            uint32_t ah[4], al[4];
            split(xr[s * 8], ah[0], al[0]);
            split(xr[s * 8 + 8 * xp], ah[1], al[1]);
            split(xr[s * 8 + 4], ah[2], al[2]);
            split(xr[s * 8 + 4 + 8 * xp], ah[3], al[3]);
            float b0[4], b1[4];
            if (DX) {                                       // tile j, column n = g: W row 8j + g
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    b0[j] = rows[(j * 8 + g) * PITCH + s * 8 + t];
                    b1[j] = rows[(j * 8 + g) * PITCH + s * 8 + t + 4];
                }
            } else if (!VEC) {                              // tile j, column n = g: W column 8j + g
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    b0[j] = rows[(s * 8 + t) * PITCH + j * 8 + g];
                    b1[j] = rows[(s * 8 + t + 4) * PITCH + j * 8 + g];
                }
            } else {                                        // tile j, column n = g: W column 4g + j, four tiles in one read
                const float4 v0 = *reinterpret_cast<const float4 *>(slot + (s * 8 + t) * PITCH + g * 4);
                const float4 v1 = *reinterpret_cast<const float4 *>(slot + (s * 8 + t + 4) * PITCH + g * 4);
                b0[0] = v0.x; b0[1] = v0.y; b0[2] = v0.z; b0[3] = v0.w;
                b1[0] = v1.x; b1[1] = v1.y; b1[2] = v1.z; b1[3] = v1.w;
            }
            mma_split(acc, ah, al, b0, b1);
        }
        if ((b + 1) % (kFlush / 32) == 0 || b + 1 == nb) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) { sum[j][e] += acc[j][e]; acc[j][e] = 0.f; }
        }
    }
    cp_async_wait<0>();
    __syncthreads();                                        // the ring is free: it takes the block's sums
    float *sums = ring;                                     // [WK][kRows][SUM_PITCH]
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float *row = sums + (kw * kRows + g + 8 * h) * SUM_PITCH + ow * 32;
        if (DX || !VEC) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float2 *>(row + j * 8 + 2 * t) = make_float2(sum[j][2 * h], sum[j][2 * h + 1]);
        } else {
            *reinterpret_cast<float4 *>(row + 8 * t) = make_float4(sum[0][2 * h], sum[1][2 * h], sum[2][2 * h], sum[3][2 * h]);
            *reinterpret_cast<float4 *>(row + 8 * t + 4) =
                make_float4(sum[0][2 * h + 1], sum[1][2 * h + 1], sum[2][2 * h + 1], sum[3][2 * h + 1]);
        }
    }
    const int ranks = static_cast<int>(gridDim.y);
    if (WK > 1) {                                           // the warps of a strip first, into the first one's place
        __syncthreads();
        for (int i = threadIdx.x; i < kRows * (OUTS / 4); i += kThreads) {
            float4 *at = reinterpret_cast<float4 *>(sums + (i / (OUTS / 4)) * SUM_PITCH + (i % (OUTS / 4)) * 4);
            float4 v = *at;
#pragma unroll
            for (int k = 1; k < WK; ++k) {
                const float4 p = at[k * kRows * SUM_PITCH / 4];
                v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
            }
            *at = v;
        }
    }
    if (ranks > 1) cluster_sync_all();
    else __syncthreads();
    for (int i = static_cast<int>(blockIdx.y) * kThreads + threadIdx.x; i < M * (OUTS / 4); i += ranks * kThreads) {
        const int m = i / (OUTS / 4), q = (i - m * (OUTS / 4)) * 4;
        const long long o = static_cast<long long>(blockIdx.x) * OUTS + q;
        if (o >= outs) continue;
        const float *at = sums + m * SUM_PITCH + q;
        const float4 v = ranks > 1 ? cluster_sum_f4(at, ranks) : *reinterpret_cast<const float4 *>(at);
        float out[4] = {v.x, v.y, v.z, v.w};
        float *dst = y + m * ldy + o;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (o + e >= outs) continue;
            if (bias) out[e] += __ldg(bias + o + e);
            if (accumulate) out[e] += dst[e];
        }
        if (y_vec && o + 3 < outs) {
            *reinterpret_cast<float4 *>(dst) = make_float4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (o + e < outs) dst[e] = out[e];
        }
    }
    if (ranks > 1) cluster_sync_all();                      // no block leaves while its sums may still be read
}

bool aligned(const void *p, size_t bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

// How a product is cut: strips of 128 outputs, or of 32 where those leave most SMs without a block; slices of at least 64
// (256 where four warps share one), at most kMaxSlices of them, as many as finish first on two blocks per SM (a block costs
// about 64 elements more than its slice).  With x staged whole and slices for two blocks per SM on average, 9 rows x 5488 x
// 7656 ran one block per SM, a few of them in a third round: forward 72.6 -> 47 us, dx 78.6 -> 44.
struct RowsPlan { int outs, k_per; unsigned strips, slices; };
RowsPlan plan_rows(int64_t outs, int64_t total, int sm_count) {
    RowsPlan p{};
    p.outs = (outs + 127) / 128 * kMaxSlices >= sm_count ? 128 : 32;
    const int64_t strips = (outs + p.outs - 1) / p.outs;
    const int64_t most = std::min<int64_t>(kMaxSlices, std::max<int64_t>(1, total / (p.outs == 128 ? 64 : 256)));
    int64_t best = 0;
    for (int64_t n = 1; n <= most; ++n) {
        const int64_t k_per = ((total + n - 1) / n + 31) / 32 * 32, slices = (total + k_per - 1) / k_per;
        const int64_t per_sm = p.outs == 128 || k_per <= 512 ? 2 : 1;
        const int64_t cost = ((strips * slices + per_sm * sm_count - 1) / (per_sm * sm_count)) * per_sm * (k_per + 64);
        if (best != 0 && cost >= best) continue;
        best = cost;
        p.k_per = static_cast<int>(k_per);
        p.slices = static_cast<unsigned>(slices);
    }
    p.strips = static_cast<unsigned>(strips);
    return p;
}

template <bool DX>
int launch_rows(const float *x, int64_t ldx, const float *W, int64_t ldw, float *y, int64_t ldy, const float *bias,
                bool accumulate, int64_t M, int64_t outs, int64_t total, int64_t w_cols, int sm_count, cudaStream_t stream) {
    const RowsPlan pl = plan_rows(outs, total, sm_count);
    const int k_per = pl.k_per;
    const bool vec = aligned(W, 16) && ldw % 4 == 0 && w_cols % 4 == 0, narrow = pl.outs == 32;
    const int x_floats = k_per <= 512 ? k_per + 4 : 2 * ((narrow ? kChunkNarrow : kChunk) + 4);
    const size_t smem = (static_cast<size_t>(kRows) * x_floats + static_cast<size_t>(kWarps) * kDepth * 32 * (DX ? 36 : 40)) * sizeof(float);
    auto kernel = narrow ? (vec ? rows_kernel<DX, true, kWarps> : rows_kernel<DX, false, kWarps>)
                         : (vec ? rows_kernel<DX, true, 1> : rows_kernel<DX, false, 1>);
    static std::atomic<uint64_t> opted_in[2][2];            // per device, as in launch_variant of the tensor path
    std::atomic<uint64_t> &done = opted_in[narrow][vec];
    int dev = 0;
    MNI_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if ((done.load(std::memory_order_acquire) & bit) == 0) {
        MNI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        done.fetch_or(bit, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pl.strips, pl.slices);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = 1;
    attrs[1].val.clusterDim.y = pl.slices;
    attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = pl.slices > 1 ? 2 : 1;
    const int y_vec = ldy % 4 == 0 && aligned(y, 16) ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, x, static_cast<long long>(ldx), W, static_cast<long long>(ldw), y,
                                             static_cast<long long>(ldy), bias, accumulate ? 1 : 0, static_cast<int>(M),
                                             static_cast<long long>(outs), static_cast<long long>(total), k_per, y_vec);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "rows_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("rows_kernel");
    return MNI_B200_OK;
}

}  // namespace

// The streaming kernel wins where its blocks cover the chip in 128-wide strips, or where the contraction is short enough
// for the 32-wide ones (measured against the tensor path, 9 rows: 4096 x 4096 18.0 / 20.1 us, 512 x 8192 6.7 / 10.3,
// 600 x 601 6.2 / 11.9; but 8192 x 512 17.4 / 13.5, 8190 x 1030 41 / 32).
bool rows_supported(int64_t M, int64_t outs, int64_t total, int sm_count) {
    return M >= 1 && M <= kRows && total >= 1 && total <= kMaxTotal && outs >= 1 &&
           outs <= 0x7fffffffLL && ((outs + 127) / 128 * kMaxSlices >= sm_count || total <= 1024);
}

int launch_rows_fwd(const float *x, int64_t ldx, const float *W, int64_t ldw, float *y, int64_t ldy, const float *bias,
                    bool accumulate, int64_t M, int64_t N, int64_t K, int sm_count, cudaStream_t stream) {
    return launch_rows<false>(x, ldx, W, ldw, y, ldy, bias, accumulate, M, N, K, N, sm_count, stream);
}
// ... with the weight stored [N, K] and seen through a transposing view
int launch_rows_bt_fwd(const float *x, int64_t ldx, const float *W, int64_t ldw, float *y, int64_t ldy, const float *bias,
                       bool accumulate, int64_t M, int64_t N, int64_t K, int sm_count, cudaStream_t stream) {
    return launch_rows<true>(x, ldx, W, ldw, y, ldy, bias, accumulate, M, N, K, K, sm_count, stream);
}
int launch_rows_dx(const float *dy, int64_t lddy, const float *W, int64_t ldw, float *dx, int64_t lddx, const float *bias,
                   bool accumulate, int64_t M, int64_t N, int64_t K, int sm_count, cudaStream_t stream) {
    return launch_rows<true>(dy, lddy, W, ldw, dx, lddx, bias, accumulate, M, K, N, N, sm_count, stream);
}
int launch_rows_bt_dx(const float *dy, int64_t lddy, const float *W, int64_t ldw, float *dx, int64_t lddx, const float *bias,
                      bool accumulate, int64_t M, int64_t N, int64_t K, int sm_count, cudaStream_t stream) {
    return launch_rows<false>(dy, lddy, W, ldw, dx, lddx, bias, accumulate, M, K, N, K, sm_count, stream);
}

}  // namespace mni
