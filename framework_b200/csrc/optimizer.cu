// The consumers of the weight gradients: global gradient norm, clip and AdamW over a list of parameters
// (ops/optimizer.rs:67-171, :247-276; kernels/adamw.cu).
//
// HBM-bound: the step reads grad and reads and writes param, m and v once (28 bytes per element), the norm reads grad
// once more.  A model's parameters are a list of tensors from a few hundred elements to millions, so the unit of work
// is a chunk of whichever tensor: ONE launch covers up to kMaxList tensors, whose addresses travel as
// a kernel parameter, and a block finds its chunk's tensor by bisection over the chunk offsets (constant memory).
// 74 tensors, 42.5 M elements: 222 launches and 1158 us a step before, of which the device worked ~400.
#include "internal.h"

#include <string.h>

#include <algorithm>
#include <iterator>
#include <map>
#include <vector>

namespace mni {

namespace {

constexpr int kThreads = 256;
constexpr int kChunk = 4096;                 // elements per block of the norm
// Elements per block of the step.  A list: four vectors of each array per thread, which pay for finding the block's tensor (74
// tensors, 42.5 M elements: 221 us; 226 with one vector).  A single tensor: one, as what such a call waits for is a block's
// later vectors (65 536 elements 7.8 us against 3.4) or a nearly empty third round of blocks (5 M 25.2 / 19.8; 50 M 224 / 215).
__host__ __device__ constexpr int step_chunk(int cap) { return cap == 1 ? 1024 : 4096; }
constexpr int kMaxList = 512;                // tensors per launch (24 KB of kernel parameters at most)
constexpr int kMaxNormBlocks = 1024;

// One entry per tensor.  first[i] = index of its first chunk; first[count] = number of chunks.
template <int CAP>
struct StepList {
    float *param[CAP], *m[CAP], *v[CAP], *grad[CAP];
    long long n[CAP];
    unsigned first[CAP + 1];
    int count;
};
template <int CAP>
struct NormList {
    const float *grad[CAP];
    long long n[CAP];
    unsigned first[CAP + 1];
    int count;
};

__device__ __forceinline__ int find_tensor(const unsigned *first, int count, unsigned chunk) {
    int lo = 0, hi = count;                  // first[lo] <= chunk < first[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= chunk) lo = mid; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void adamw_one(float &p, float &m, float &v, float g, const AdamWArgs &a) {
    const float mi = a.beta1 * m + (1.0f - a.beta1) * g;
    const float vi = a.beta2 * v + (1.0f - a.beta2) * g * g;
    m = mi;
    v = vi;
    p = p * a.decay - a.lr * (mi / a.bc1) / (sqrtf(vi / a.bc2) + a.eps);
}
// Clip factor of ops/optimizer.rs:232-236: max_norm / norm when the norm (f64 sum of squares, rounded to
// f32, then sqrt) exceeds max_norm, else 1.  The sum of squares is read from device memory, so no
// host round trip sits between the norm and the step.
__device__ __forceinline__ float clip_scale(const double *sumsq, float max_norm) {
    if (sumsq == nullptr || !(max_norm > 0.0f)) return 1.0f;
    const float norm = sqrtf(static_cast<float>(*static_cast<const volatile double *>(sumsq)));
    return norm > max_norm ? max_norm / norm : 1.0f;
}

// One block per chunk, last chunk first: the norm kernel before it read the gradients in ascending order, so the
// ones it read last are still in L2.  Launched as a dependent of the norm kernel: everything but the norm itself is
// fetched before the wait (the norm kernel was launched the ordinary way, so whatever wrote the operands is complete
// once it runs).
template <int CAP>
__global__ void __launch_bounds__(kThreads, CAP == 1 ? 6 : 4)
adamw_list_kernel(const __grid_constant__ StepList<CAP> list, const AdamWArgs a) {
    constexpr int CHUNK = step_chunk(CAP);
    const unsigned chunk = list.first[list.count] - 1 - blockIdx.x;
    const int t = find_tensor(list.first, list.count, chunk);
    const long long base = static_cast<long long>(chunk - list.first[t]) * CHUNK, n = list.n[t];
    float *param = list.param[t], *m = list.m[t], *v = list.v[t], *grad = list.grad[t];
    const bool vec = ((reinterpret_cast<uintptr_t>(param) | reinterpret_cast<uintptr_t>(m) |
                       reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(grad)) & 15) == 0;
    float scale = 1.0f;
    if (vec && base + CHUNK <= n) {
        constexpr int PER = CHUNK / (kThreads * 4), U = PER < 2 ? PER : 2;
#pragma unroll
        for (int h = 0; h < PER / U; ++h) {
            float4 p[U], mm[U], vv[U], g[U];
            long long at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                at[u] = base + ((h * U + u) * kThreads + threadIdx.x) * 4;
                p[u] = *reinterpret_cast<const float4 *>(param + at[u]);
                mm[u] = *reinterpret_cast<const float4 *>(m + at[u]);
                vv[u] = *reinterpret_cast<const float4 *>(v + at[u]);
                g[u] = __ldcs(reinterpret_cast<const float4 *>(grad + at[u]));
            }
            if (h == 0) {
                grid_dependency_wait();
                scale = clip_scale(a.sumsq, a.max_norm);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (scale != 1.0f) {
                    g[u].x *= scale; g[u].y *= scale; g[u].z *= scale; g[u].w *= scale;
                    if (a.write_grad) *reinterpret_cast<float4 *>(grad + at[u]) = g[u];
                }
                adamw_one(p[u].x, mm[u].x, vv[u].x, g[u].x, a);
                adamw_one(p[u].y, mm[u].y, vv[u].y, g[u].y, a);
                adamw_one(p[u].z, mm[u].z, vv[u].z, g[u].z, a);
                adamw_one(p[u].w, mm[u].w, vv[u].w, g[u].w, a);
                *reinterpret_cast<float4 *>(param + at[u]) = p[u];
                *reinterpret_cast<float4 *>(m + at[u]) = mm[u];
                *reinterpret_cast<float4 *>(v + at[u]) = vv[u];
            }
        }
        return;
    }
    // A tensor's last, partial chunk, or one that is not 16-byte aligned: four elements of each array of a thread on their way
    // together (one after the other they cost a round trip to memory each: 3100 elements 11.6 us, now 3.0).
    const long long end = min(n, base + CHUNK);
#pragma unroll 1
    for (int h = 0; h < CHUNK; h += 4 * kThreads) {
        const long long i0 = base + h + threadIdx.x;
        float p[4], mm[4], vv[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * kThreads;
            if (i >= end) continue;
            p[u] = param[i]; mm[u] = m[i]; vv[u] = v[i];
            g[u] = __ldcs(grad + i);
        }
        if (h == 0) {
            grid_dependency_wait();
            scale = clip_scale(a.sumsq, a.max_norm);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * kThreads;
            if (i >= end) continue;
            if (scale != 1.0f) {
                g[u] *= scale;
                if (a.write_grad) grad[i] = g[u];
            }
            adamw_one(p[u], mm[u], vv[u], g[u], a);
            param[i] = p[u]; m[i] = mm[u]; v[i] = vv[u];
        }
        if (i0 + 4 * kThreads - threadIdx.x >= end) break;
    }
}

// ---- gradient norm (ops/optimizer.rs:126-138): f64 sum of f32 squares ------------------------------
// A grid of at most kMaxNormBlocks blocks walks the chunks; every thread keeps an f64 sum, every block adds its
// threads in a fixed order, and the block that takes the last ticket adds the blocks' sums in a fixed order.  The
// grid depends on the sizes and the SM count only, so the result is reproducible run to run.
__device__ double g_norm_partial[kMaxNormBlocks];
__device__ unsigned g_norm_ticket;           // zero between launches
__device__ double g_norm_sumsq;              // clip_and_step's squared norm

__device__ __forceinline__ double block_sum_f64(double x) {
    __shared__ double warp_sums[kThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    __syncthreads();                          // warp_sums may still be read from the last call
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kThreads / 32; ++w) t += warp_sums[w];
    return t;   // valid in thread 0
}
__device__ __forceinline__ void add_squares(double &acc, const float4 &t) {
    acc += static_cast<double>(t.x) * t.x;
    acc += static_cast<double>(t.y) * t.y;
    acc += static_cast<double>(t.z) * t.z;
    acc += static_cast<double>(t.w) * t.w;
}
// out (device) receives the sum; `slot` (pinned host memory, may be null) receives it too, followed by slot->seq.
template <int CAP>
__global__ void __launch_bounds__(kThreads)
sumsq_list_kernel(const __grid_constant__ NormList<CAP> list, double *out, int accumulate, NormSlot *slot, unsigned seq) {
    grid_dependency_trigger();
    __shared__ bool s_last;
    double acc = 0.0, acc2 = 0.0;
    const unsigned chunks = list.first[list.count];
    for (unsigned chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
        const int t = find_tensor(list.first, list.count, chunk);
        const long long base = static_cast<long long>(chunk - list.first[t]) * kChunk, n = list.n[t];
        const float *g = list.grad[t];
        if ((reinterpret_cast<uintptr_t>(g) & 15) == 0 && base + kChunk <= n) {
            constexpr int U = kChunk / (kThreads * 4);
            float4 x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) x[u] = *reinterpret_cast<const float4 *>(g + base + (u * kThreads + threadIdx.x) * 4);
#pragma unroll
            for (int u = 0; u < U; ++u) add_squares((u & 1) ? acc2 : acc, x[u]);
        } else {
            const long long end = min(n, base + kChunk);
            for (long long i = base + threadIdx.x; i < end; i += kThreads) acc += static_cast<double>(g[i]) * g[i];
        }
    }
    const double t = block_sum_f64(acc + acc2);
    if (threadIdx.x == 0) {
        g_norm_partial[blockIdx.x] = t;
        __threadfence();
        s_last = atomicAdd(&g_norm_ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double sum = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += kThreads) sum += __ldcg(g_norm_partial + i);
    sum = block_sum_f64(sum);
    if (threadIdx.x == 0) {
        if (accumulate) sum += *out;
        *out = sum;
        g_norm_ticket = 0u;
        if (slot) {
            slot->sumsq = sum;
            __threadfence_system();
            *static_cast<volatile unsigned *>(&slot->seq) = seq;
        }
    }
}

unsigned chunks_of(int64_t n, int chunk) { return static_cast<unsigned>((n + chunk - 1) / chunk); }

template <int CAP>
int launch_step(const AdamWArgs &a, int count, float *const *param, float *const *m, float *const *v, float *const *grad,
                const int64_t *n, bool dependent, cudaStream_t stream) {
    StepList<CAP> list;
    list.count = 0;
    list.first[0] = 0;
    for (int i = 0; i < count; ++i) {
        if (n[i] == 0) continue;
        const int k = list.count++;
        list.param[k] = param[i]; list.m[k] = m[i]; list.v[k] = v[i]; list.grad[k] = grad[i];
        list.n[k] = n[i];
        list.first[k + 1] = list.first[k] + chunks_of(n[i], step_chunk(CAP));
    }
    if (list.count == 0) return MNI_B200_OK;
    const dim3 grid(list.first[list.count]), block(kThreads);
    if (dependent) {
        const cudaError_t e = launch_dependent(adamw_list_kernel<CAP>, grid, block, 0, stream, list, a);
        if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "adamw launch failed: %s", cudaGetErrorString(e));
    } else {
        adamw_list_kernel<CAP><<<grid, block, 0, stream>>>(list, a);
    }
    MNI_LAUNCH_CHECK("adamw_list_kernel");
    return MNI_B200_OK;
}

template <int CAP>
int launch_norm(int count, const float *const *grad, const int64_t *n, double *out, bool accumulate, NormSlot *slot,
                unsigned seq, int sm_count, cudaStream_t stream) {
    NormList<CAP> list;
    list.count = 0;
    list.first[0] = 0;
    for (int i = 0; i < count; ++i) {
        if (n[i] == 0) continue;
        const int k = list.count++;
        list.grad[k] = grad[i];
        list.n[k] = n[i];
        list.first[k + 1] = list.first[k] + chunks_of(n[i], kChunk);
    }
    const unsigned chunks = list.first[list.count];
    const unsigned blocks = std::max(1u, std::min(chunks, static_cast<unsigned>(std::min(6 * sm_count, kMaxNormBlocks))));
    sumsq_list_kernel<CAP><<<blocks, kThreads, 0, stream>>>(list, out, accumulate ? 1 : 0, slot, seq);
    MNI_LAUNCH_CHECK("sumsq_list_kernel");
    return MNI_B200_OK;
}

// Memory that the step of entry `entry` writes.
struct Span { uintptr_t begin, end; int64_t entry; };

// Whether the steps of two entries touch the same memory.  A model's tensors mostly come in the order of their addresses, each
// kind in a buffer of its own, where one look at each settles it; or else as four sorted runs that only need merging.  (The
// kernel of a short list's norm is over in 5 us, and the step is launched behind this check.)
bool entries_overlap(int64_t count, float *const *const (&arrays)[4], const int64_t *n) {
    Span range[4];
    bool settled = true;
    for (int k = 0; k < 4 && settled; ++k) {
        range[k] = Span{0, 0, -1};
        for (int64_t i = 0; i < count && settled; ++i) {
            if (n[i] == 0) continue;
            const uintptr_t at = reinterpret_cast<uintptr_t>(arrays[k][i]);
            settled = at >= range[k].end;
            if (range[k].entry < 0) range[k].begin = at;
            range[k].end = at + static_cast<uintptr_t>(n[i]) * sizeof(float);
            range[k].entry = i;
        }
        for (int j = 0; j < k && settled; ++j) settled = range[k].begin >= range[j].end || range[j].begin >= range[k].end;
    }
    if (settled) return false;
    std::vector<Span> spans;
    spans.reserve(static_cast<size_t>(4 * count));
    auto less = [](const Span &a, const Span &b) { return a.begin < b.begin; };
    std::ptrdiff_t runs[5] = {0, 0, 0, 0, 0};
    for (int k = 0; k < 4; ++k) {
        for (int64_t i = 0; i < count; ++i) {
            const uintptr_t at = reinterpret_cast<uintptr_t>(arrays[k][i]);
            if (n[i] > 0) spans.push_back(Span{at, at + static_cast<uintptr_t>(n[i]) * sizeof(float), i});
        }
        runs[k + 1] = static_cast<std::ptrdiff_t>(spans.size());
        const auto first = spans.begin() + runs[k];
        if (!std::is_sorted(first, spans.end(), less)) std::sort(first, spans.end(), less);
    }
    const auto at = spans.begin();
    std::inplace_merge(at, at + runs[1], at + runs[2], less);
    std::inplace_merge(at + runs[2], at + runs[3], at + runs[4], less);
    std::inplace_merge(at, at + runs[2], at + runs[4], less);
    Span reach{0, 0, -1};
    for (const Span &s : spans) {
        if (s.begin < reach.end && s.entry != reach.entry) return true;
        if (s.end > reach.end) reach = s;
    }
    return false;
}

// How many entries from the start of the list one launch may take: up to the first that touches what an earlier one writes.
int64_t disjoint_entries(int64_t count, float *const *const (&arrays)[4], const int64_t *n) {
    std::map<uintptr_t, uintptr_t> taken;                     // begin -> end, disjoint
    for (int64_t i = 0; i < count; ++i) {
        if (n[i] == 0) continue;
        Span own[4];
        for (int k = 0; k < 4; ++k) {
            const uintptr_t at = reinterpret_cast<uintptr_t>(arrays[k][i]);
            own[k] = Span{at, at + static_cast<uintptr_t>(n[i]) * sizeof(float), i};
        }
        std::sort(own, own + 4, [](const Span &a, const Span &b) { return a.begin < b.begin; });
        int parts = 1;                                        // an entry's own arrays may overlap
        for (int k = 1; k < 4; ++k) {
            if (own[k].begin < own[parts - 1].end) own[parts - 1].end = std::max(own[parts - 1].end, own[k].end);
            else own[parts++] = own[k];
        }
        for (int k = 0; k < parts; ++k) {
            const auto next = taken.upper_bound(own[k].begin);
            if (next != taken.end() && next->first < own[k].end) return i;
            if (next != taken.begin() && std::prev(next)->second > own[k].begin) return i;
        }
        for (int k = 0; k < parts; ++k) taken[own[k].begin] = own[k].end;
    }
    return count;
}

}  // namespace

double *norm_sumsq_ptr() {
    void *p = nullptr;
    return cudaGetSymbolAddress(&p, g_norm_sumsq) == cudaSuccess ? static_cast<double *>(p) : nullptr;
}

// Entries that touch the same memory (tied parameters given twice) are stepped one after the other, in list order: the blocks of
// one launch run in any order, so a launch ends before an entry that overlaps one of its own.
int launch_adamw_list(const AdamWArgs &a, int64_t count, float *const *param, float *const *m, float *const *v,
                      float *const *grad, const int64_t *n, bool dependent, cudaStream_t stream) {
    float *const *const arrays[4] = {param, m, v, grad};
    const bool overlap = count > 1 && entries_overlap(count, arrays, n);
    for (int64_t i = 0, k64 = 0; i < count; i += k64) {
        k64 = std::min<int64_t>(kMaxList, count - i);
        if (overlap) {
            float *const *const rest[4] = {param + i, m + i, v + i, grad + i};
            k64 = disjoint_entries(k64, rest, n + i);
        }
        const int k = static_cast<int>(k64);
        // the parameter block is copied at every launch, so a short list takes a short one
        auto launch = k == 1 ? launch_step<1> : k <= 16 ? launch_step<16> : k <= 128 ? launch_step<128> : launch_step<kMaxList>;
        const int rc = launch(a, k, param + i, m + i, v + i, grad + i, n + i, dependent && i == 0, stream);
        if (rc) return rc;
    }
    return MNI_B200_OK;
}

int launch_sumsq_list(int64_t count, const float *const *grad, const int64_t *n, double *out, bool accumulate,
                      NormSlot *slot, unsigned seq, int sm_count, cudaStream_t stream) {
    for (int64_t i = 0; i == 0 || i < count; i += kMaxList) {
        const int k = static_cast<int>(std::min<int64_t>(kMaxList, count - i));
        const bool last = i + kMaxList >= count;
        auto launch = k <= 16 ? launch_norm<16> : k <= 128 ? launch_norm<128> : launch_norm<kMaxList>;
        const int rc = launch(k, grad + i, n + i, out, accumulate || i > 0, last ? slot : nullptr, seq, sm_count, stream);
        if (rc) return rc;
    }
    return MNI_B200_OK;
}

}  // namespace mni
