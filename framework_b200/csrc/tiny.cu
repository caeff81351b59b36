// Products too small for the tensor path: plain f32 on the FMA units, all products of a call (and its column sums) in one
// launch.  At these sizes a tensor-path launch is its fixed chain -- barriers, tensor memory, descriptor fetch, TMA round
// trip, split, MMA, commit, TMEM load, staging, TMA store: 4.6-5.8 us for one k-block -- and a backward call is three
// launches on two streams.  Here a block's loads are issued at once and the arithmetic is a few hundred cycles:
// 32 x 64 x 32 forward 4.3 -> 2.8 us, backward with the bias gradient 6.1 -> 2.6; 128^3 5.9 -> 4.0 and 9.4 -> 4.0.
//
// A block owns a 32 x 32 tile of one product.  Its eight warps take every eighth run of 8 contraction elements, each
// with a private slice of shared memory (no barrier in the loop) and the next run's loads in registers while the current
// one is multiplied: a lane keeps 8 x 4 outputs, so three 16-byte reads feed 32 FMAs.  The warps' sums are added in warp
// order: results do not depend on scheduling.
//
// Its stores are single elements and a tile's 256 threads take a slot whatever the tile holds, so it is for calls of few tiles:
// api.cu has the limits.
#include "activation.h"
#include "internal.h"

#include <algorithm>

namespace mni {

namespace {

constexpr int kWarps = 8;
constexpr int kThreads = 32 * kWarps;
constexpr int kTile = 32, kRun = 8;          // tile edge, contraction elements of a warp's step
constexpr int kPitch = kTile + 4;

struct Job {
    TinyProduct p;
    int tiles_n;
    unsigned first;                          // first block
};
struct Jobs {
    Job job[kMaxTiny];
    TinyColumns columns;                     // column sums, after the products' blocks
    unsigned columns_first;
    int count;
};

// What a lane loads of an operand tile in one step: eight elements `step` apart from `ptr`, consecutive lanes along the
// dimension of unit stride (k_unit: 8 lanes along k, rows 4 apart; otherwise 32 lanes along the rows, k next to each other).
// Their places in shared memory are `pitch` apart from `slot`.
struct Lane {
    const float *ptr;
    long long step, advance;                 // ... and to the same element of the warp's next step
    int slot, pitch, k;                      // k: of the first element
    unsigned rows;                           // bit i: element i's row exists
    bool k_unit;
};
__device__ __forceinline__ Lane make_lane(const float *ptr, long long s_row, long long s_k, int row0, int rows, int lane, int warp) {
    Lane l;
    l.k_unit = s_k == 1 && s_row != 1;
    const int r = l.k_unit ? lane >> 3 : lane, k = warp * kRun + (l.k_unit ? lane & 7 : 0);
    l.ptr = ptr + (row0 + r) * s_row + k * s_k;
    l.step = l.k_unit ? 4 * s_row : s_k;
    l.advance = kRun * kWarps * s_k;
    l.k = k;
    l.slot = (l.k_unit ? lane & 7 : 0) * kPitch + r;
    l.pitch = l.k_unit ? 4 : kPitch;
    l.rows = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (row0 + r + (l.k_unit ? 4 * i : 0) < rows) l.rows |= 1u << i;
    return l;
}
__device__ __forceinline__ void load_step(Lane &l, int K, float (&v)[8]) {
    // k_unit: one k for all eight; otherwise k, k + 1, ...
    const int left = K - l.k;
    const unsigned ok = l.rows & (l.k_unit ? (left > 0 ? 0xffu : 0u) : (left >= 8 ? 0xffu : left > 0 ? (1u << left) - 1u : 0u));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = 0.f;
        if (ok >> i & 1u) v[i] = __ldg(l.ptr + i * l.step);
    }
    l.ptr += l.advance;
    l.k += kRun * kWarps;
}

// ACT: the products are followed by bias + GELU (its registers cost the others 0.5 us in 6).
template <bool ACT>
__global__ void __launch_bounds__(kThreads)
tiny_kernel(const __grid_constant__ Jobs jobs) {
    __shared__ __align__(16) float mem[kWarps * kTile * kPitch];     // operand slices [warp][2][kRun][kPitch], then the sums
    grid_dependency_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x >= jobs.columns_first) {
        const TinyColumns &c = jobs.columns;
        const int col = static_cast<int>(blockIdx.x - jobs.columns_first) * 32 + lane;
        grid_dependency_wait();
        float s = 0.f;
        if (col < c.n) {
#pragma unroll 8
            for (int r = warp; r < c.rows; r += kWarps) s += __ldg(c.src + static_cast<long long>(r) * c.ld + col);
        }
        mem[warp * 32 + lane] = s;
        __syncthreads();
        if (warp == 0 && col < c.n) {
            float t = mem[lane];
#pragma unroll
            for (int w = 1; w < kWarps; ++w) t += mem[w * 32 + lane];
            c.out[col] = c.accumulate ? c.out[col] + t : t;
        }
        return;
    }
    int j = 0;
    while (j + 1 < jobs.count && blockIdx.x >= jobs.job[j + 1].first) ++j;
    const TinyProduct &p = jobs.job[j].p;
    const int tile = static_cast<int>(blockIdx.x - jobs.job[j].first);
    const int m0 = tile / jobs.job[j].tiles_n * kTile, n0 = tile % jobs.job[j].tiles_n * kTile;
    float *sa = mem + warp * (2 * kRun * kPitch), *sb = sa + kRun * kPitch;
    Lane la = make_lane(p.a, p.a_m, p.a_k, m0, p.M, lane, warp), lb = make_lane(p.b, p.b_n, p.b_k, n0, p.N, lane, warp);
    const int K = p.K;
    float ra[8], rb[8];
    grid_dependency_wait();
    const int r0 = (lane >> 3) * 8, c0 = (lane & 7) * 4;
    float acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
    load_step(la, K, ra);
    load_step(lb, K, rb);
    for (int k0 = warp * kRun; k0 < K; k0 += kRun * kWarps) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            sa[la.slot + i * la.pitch] = ra[i];
            sb[lb.slot + i * lb.pitch] = rb[i];
        }
        __syncwarp();
        load_step(la, K, ra);                               // past the end: nothing is read
        load_step(lb, K, rb);
#pragma unroll
        for (int k = 0; k < kRun; ++k) {
            const float4 a0 = *reinterpret_cast<const float4 *>(sa + k * kPitch + r0);
            const float4 a1 = *reinterpret_cast<const float4 *>(sa + k * kPitch + r0 + 4);
            const float4 b = *reinterpret_cast<const float4 *>(sb + k * kPitch + c0);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r], bv[c], acc[r][c]);
        }
        __syncwarp();
    }
    __syncthreads();                                        // the slices are free: they take the warps' sums
    float *sums = mem + warp * (kTile * kPitch);
#pragma unroll
    for (int r = 0; r < 8; ++r)
        *reinterpret_cast<float4 *>(sums + (r0 + r) * kPitch + c0) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    __syncthreads();
    const int row = threadIdx.x >> 3, col = (threadIdx.x & 7) * 4;
    if (m0 + row >= p.M || n0 + col >= p.N) return;
    float4 s = *reinterpret_cast<const float4 *>(mem + row * kPitch + col);
    const int live = min(kWarps, (K + kRun - 1) / kRun);
    for (int w = 1; w < live; ++w) {
        const float4 t = *reinterpret_cast<const float4 *>(mem + w * (kTile * kPitch) + row * kPitch + col);
        s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
    }
    float out[4] = {s.x, s.y, s.z, s.w};
    const long long at = (m0 + row) * p.ldc + n0 + col;
    float *dst = p.c + at;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (n0 + col + e >= p.N) break;
        if (ACT) {
            if (p.c) dst[e] = out[e];
            p.act[at + e] = gelu_tanh(out[e] + __ldg(p.bias + n0 + col + e));
            continue;
        }
        if (p.bias) out[e] += __ldg(p.bias + n0 + col + e);
        if (p.accumulate) out[e] += dst[e];
        dst[e] = out[e];
    }
}

}  // namespace

int launch_tiny(const TinyProduct *products, int count, const TinyColumns *columns, cudaStream_t stream) {
    Jobs jobs;
    jobs.count = count;
    unsigned blocks = 0;
    for (int i = 0; i < count; ++i) {
        Job &j = jobs.job[i];
        j.p = products[i];
        j.first = blocks;
        j.tiles_n = (products[i].N + kTile - 1) / kTile;
        blocks += static_cast<unsigned>((products[i].M + kTile - 1) / kTile * j.tiles_n);
    }
    jobs.columns_first = blocks;
    jobs.columns = TinyColumns{};
    if (columns) {
        jobs.columns = *columns;
        blocks += static_cast<unsigned>((columns->n + 31) / 32);
    }
    if (blocks == 0) return MNI_B200_OK;
    const cudaError_t e = launch_dependent(products[0].act ? tiny_kernel<true> : tiny_kernel<false>, dim3(blocks), dim3(kThreads), 0, stream, jobs);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "tiny_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("tiny_kernel");
    return MNI_B200_OK;
}

}  // namespace mni
