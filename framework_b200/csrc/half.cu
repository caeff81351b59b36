// Operands of large products in 16-bit planes for the f16 tensor pipe, which runs at twice the rate of TF32 and has the same
// eleven significant bits: x * 2^e = hi + lo * 2^-12 with hi and lo in f16, e chosen for the whole operand.
//
// e comes from 1024 sampled elements, so one pass over the operand is enough; the largest sample lands in [2^6, 2^7).  Above it
// there is room for elements 256 times as large, below it every element of at least 2^-14, which is 2^-20 of it or less, keeps 22
// bits (11 where there is no lo).  What f16 does not hold is found by the same pass and reported in the block's status word; a
// second kernel then writes three bf16 planes, whose range is that of f32, and the products take those:
//   - an element beyond 2^15 after scaling, an infinity or a NaN;
//   - a stretch of a row (256 elements) or of a column (what a block takes of it in one matrix) in which more than a fifth of the
//     elements are smaller than 2^-14, zeros not counted: in its row or column of the product the bits they lose could be the
//     leading ones, where the stretch has nothing else as well as where the rest of it meets zeros;
//   - 64 columns of what a block takes of a matrix with more than 16 small elements that are more than a sixteenth of all.
// So a small element that stays has four times as many ordinary ones beside it, in its row and in its column.  It carries an
// absolute error of 2^-43 (2^-31 without lo) of the largest sample.  Of normally distributed elements one in 6e5 is small: two of
// a stretch's first ten do not come about by chance.
#include "internal.h"

#include <cuda_fp16.h>

#include <algorithm>

namespace mni {

namespace {

constexpr int kThreads = 256, kTileRows = 16, kTileCols = 512;     // 64 threads x 8 columns, 4 groups of 4 rows
constexpr int kBlocksPerSm = 3;
constexpr float kLargest = 32768.f, kSmallest = 1.f / 16384.f;
constexpr unsigned kOrdinary = 4;                  // this many ordinary elements to each small one
constexpr int kMaxExp = kHalfMaxExp, kTargetExp = 6;
// Status word of a block: some element, row or column did not fit; some element is beyond 2^30 after scaling.
constexpr unsigned kUnfit = 1, kHuge = 2;

struct View {
    const float *src;
    uint16_t *dst;                      // first plane; the others follow `plane` elements apart
    long long ld, b0, b1, b2;           // source strides
    long long matrix, plane;
    int rows, cols, pitch;
    FastDiv rows_d, d1, d2;
    FastDiv tiles_r, tiles_strip;       // tiles of a strip of columns: of one matrix, of all of them
    int first_tile;
    unsigned total_rows;
    int vec;                            // rows are 16-byte aligned
    int *exp;
};
struct ViewList {
    View v[kMaxHalves];
    int count, tiles;
    unsigned int *status;
    int statuses;                       // = blocks of split_half_kernel
    unsigned int *verdict;              // all of them in one word, for the products
    HalfColumns sums;                   // of the first view
};

__device__ __forceinline__ const float *matrix_source(const View &v, int batch) {
    const int q2 = fd_div(batch, v.d2), q1 = fd_div(q2, v.d1);
    return v.src + (batch - q2 * static_cast<int>(v.d2.d)) * v.b2 + (q2 - q1 * static_cast<int>(v.d1.d)) * v.b1 + q1 * v.b0;
}
struct Tile {
    int strip, batch, r0, c0;           // r0: first row of the tile, c0: first column of its strip
};
__device__ __forceinline__ Tile tile_at(const View &v, int rel) {
    Tile t;
    t.strip = fd_div(rel, v.tiles_strip);
    const int in = rel - t.strip * static_cast<int>(v.tiles_strip.d);
    t.batch = fd_div(in, v.tiles_r);
    t.r0 = (in - t.batch * static_cast<int>(v.tiles_r.d)) * kTileRows;
    t.c0 = t.strip * kTileCols;
    return t;
}
__device__ __forceinline__ int first_tile_of(const ViewList &list, int block) {
    return static_cast<int>(static_cast<long long>(list.tiles) * block / list.statuses);
}

// The exponent of the operand's scale, the same in every block that asks.
__device__ int operand_exponent(const View &v, unsigned *biggest) {
    unsigned m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned s = i * kThreads + threadIdx.x;
        const int row = static_cast<int>((static_cast<unsigned long long>(s) * v.total_rows) >> 10);
        unsigned h = (s + 1u) * 0x9E3779B1u;
        h = (h ^ (h >> 15)) * 0x85EBCA77u;
        h ^= h >> 13;
        const int col = static_cast<int>(__umulhi(h, static_cast<unsigned>(v.cols)));
        const int batch = fd_div(row, v.rows_d);
        const float x = __ldg(matrix_source(v, batch) + (row - batch * v.rows) * v.ld + col);
        m = max(m, __float_as_uint(x) & 0x7fffffffu);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) biggest[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) m = max(m, biggest[w]);
    const int field = static_cast<int>(m >> 23);                    // 255: infinity or NaN, which the pass will find
    return (m == 0 || field == 255) ? 0 : max(-kMaxExp, min(kMaxExp, kTargetExp + 127 - field));
}

// Bound by memory: 4 bytes read and 4 (LO) or 2 written an element.  A block takes consecutive tiles of a strip of columns, so
// that what it finds about columns stays in registers until the matrix ends, and their sums (SUMS: of the first view, for the
// bias gradient) until the strip ends.  The ordinary elements of a column are counted two columns at a time, in f16, which stops at 2048 and so errs
// towards "unfit" only.
template <bool LO, bool SUMS>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
split_half_kernel(const __grid_constant__ ViewList list) {
    __shared__ unsigned shared[4][kTileCols];
    grid_dependency_trigger();
    grid_dependency_wait();
    const int t0 = first_tile_of(list, blockIdx.x), t1 = first_tile_of(list, blockIdx.x + 1);
    const int tc = threadIdx.x & 63, group = threadIdx.x >> 6;
    const unsigned limit = __float_as_uint(kLargest), small = __float_as_uint(kSmallest);
    const __half2 none = __float2half2_rn(0.f), least_ordinary = __float2half2_rn(kSmallest);
    unsigned bad = 0;
    __half2 ordinary[4], few[4];                   // of the columns: elements of 2^-14 and more, smaller ones but zeros
    float sum[8];
    bool some_small = false;
    int j = -1, strip = -1;
    float scale = 1.f;
    auto begin_columns = [&] {
#pragma unroll
        for (int c = 0; c < 4; ++c) ordinary[c] = few[c] = none;
        some_small = false;
    };
    auto end_columns = [&] {
        if (__syncthreads_or(some_small)) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const __half o = c & 1 ? __high2half(ordinary[c / 2]) : __low2half(ordinary[c / 2]);
                const __half f = c & 1 ? __high2half(few[c / 2]) : __low2half(few[c / 2]);
                shared[group][tc * 8 + c] = __half2uint_rz(o) | __half2uint_rz(f) << 16;
            }
            __syncthreads();
            unsigned smalls = 0, others = 0;
            for (int c = threadIdx.x; c < kTileCols; c += kThreads) {
                const unsigned n = shared[0][c] + shared[1][c] + shared[2][c] + shared[3][c];      // at most 8192 each
                if (kOrdinary * (n >> 16) > (n & 0xffffu)) bad |= kUnfit;
                smalls += n >> 16;
                others += n & 0xffffu;
            }
            smalls = __reduce_add_sync(0xffffffffu, smalls);
            others = __reduce_add_sync(0xffffffffu, others);
            if (smalls > 16 + (smalls + others) / 16) bad |= kUnfit;
        }
    };
    auto end_strip = [&] {
        end_columns();
        if (SUMS && j == 0) {
            __syncthreads();
            float *const mine = reinterpret_cast<float *>(&shared[0][0]);
#pragma unroll
            for (int c = 0; c < 8; ++c) mine[group * kTileCols + tc * 8 + c] = sum[c];
            __syncthreads();
            float *const out = list.sums.partial + static_cast<long long>(blockIdx.x + strip) * kTileCols;
            for (int c = threadIdx.x; c < kTileCols; c += kThreads)
                out[c] = (mine[c] + mine[kTileCols + c]) + (mine[2 * kTileCols + c] + mine[3 * kTileCols + c]);
            __syncthreads();
        }
    };
    for (int tile = t0; tile < t1; ++tile) {
        int at = 0;
        while (at + 1 < list.count && tile >= list.v[at + 1].first_tile) ++at;
        const View &v = list.v[at];
        const Tile t = tile_at(v, tile - v.first_tile);
        const int r0 = t.r0 + group, c0 = t.c0 + tc * 8;
        const float *src = matrix_source(v, t.batch) + r0 * v.ld + c0;
        const bool whole = v.vec && c0 + 8 <= v.cols;
        float x[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float *row = src + 4 * i * v.ld;
            if (r0 + 4 * i < v.rows && whole) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(row)), b = __ldg(reinterpret_cast<const float4 *>(row) + 1);
                x[i][0] = a.x; x[i][1] = a.y; x[i][2] = a.z; x[i][3] = a.w;
                x[i][4] = b.x; x[i][5] = b.y; x[i][6] = b.z; x[i][7] = b.w;
            } else {
#pragma unroll
                for (int c = 0; c < 8; ++c) x[i][c] = (r0 + 4 * i < v.rows && c0 + c < v.cols) ? __ldg(row + c) : 0.f;
            }
        }
        if (at != j || t.strip != strip) {         // the loads above are on their way meanwhile
            if (j >= 0) end_strip();
            if (at != j) {
                const int e = operand_exponent(v, &shared[0][0]);
                __syncthreads();
                scale = __uint_as_float(static_cast<unsigned>(127 + e) << 23);
                if (tile == v.first_tile && threadIdx.x == 0) *v.exp = e;
            }
            j = at;
            strip = t.strip;
            begin_columns();
            if (SUMS) {
#pragma unroll
                for (int c = 0; c < 8; ++c) sum[c] = 0.f;
            }
        } else if (t.r0 == 0) {                    // the next matrix, whose columns are judged by themselves
            end_columns();
            begin_columns();
        }
        uint16_t *dst = v.dst + t.batch * v.matrix + static_cast<long long>(r0) * v.pitch + c0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (r0 + 4 * i >= v.rows) break;       // the same for the whole warp
            uint4 hi, lo;
            unsigned *const h = &hi.x, *const l = &lo.x;
            unsigned big = 0, least = 0xffffffffu;
#pragma unroll
            for (int c = 0; c < 8; c += 2) {
                if (SUMS) { sum[c] += x[i][c]; sum[c + 1] += x[i][c + 1]; }
                const float a = x[i][c] * scale, b = x[i][c + 1] * scale;
                const unsigned ua = __float_as_uint(a) & 0x7fffffffu, ub = __float_as_uint(b) & 0x7fffffffu;
                big = max(big, max(ua, ub));
                least = min(least, min(ua - 1u, ub - 1u));         // a zero wraps round to the largest
                const __half2 h2 = __floats2half2_rn(a, b);
                h[c / 2] = *reinterpret_cast<const unsigned *>(&h2);
                ordinary[c / 2] = __hadd2(ordinary[c / 2], __hge2(__habs2(h2), least_ordinary));
                if (LO) {
                    const float2 back = __half22float2(h2);
                    constexpr float up = 1 << kHalfLoShift;
                    const __half2 l2 = __floats2half2_rn((a - back.x) * up, (b - back.y) * up);
                    l[c / 2] = *reinterpret_cast<const unsigned *>(&l2);
                }
            }
            if (big > limit) bad |= big > __float_as_uint(1073741824.f) ? kUnfit | kHuge : kUnfit;
            if (__any_sync(0xffffffffu, least < small - 1u)) {
                unsigned n = 0;                                    // small ones below, ordinary ones above
#pragma unroll
                for (int c = 0; c < 8; c += 2) {
                    const unsigned ua = __float_as_uint(x[i][c] * scale) & 0x7fffffffu, ub = __float_as_uint(x[i][c + 1] * scale) & 0x7fffffffu;
                    const bool sa = ua - 1u < small - 1u, sb = ub - 1u < small - 1u;
                    n += (sa ? 1u : ua ? 0x10000u : 0u) + (sb ? 1u : ub ? 0x10000u : 0u);
                    few[c / 2] = __hadd2(few[c / 2], __floats2half2_rn(sa ? 1.f : 0.f, sb ? 1.f : 0.f));
                }
                some_small = true;                                 // of the warp, that is
                n = __reduce_add_sync(0xffffffffu, n);
                if (kOrdinary * (n & 0xffffu) > n >> 16) bad |= kUnfit;
            }
            if (c0 < v.pitch) {
                *reinterpret_cast<uint4 *>(dst + static_cast<long long>(4 * i) * v.pitch) = hi;
                if (LO) *reinterpret_cast<uint4 *>(dst + v.plane + static_cast<long long>(4 * i) * v.pitch) = lo;
            }
        }
    }
    if (j >= 0) end_strip();
    bad = (__syncthreads_or(bad & kUnfit) ? kUnfit : 0u) | (__syncthreads_or(bad & kHuge) ? kHuge : 0u);
    if (threadIdx.x == 0) list.status[blockIdx.x] = bad;
}

// The bf16 of plane `plane` in the upper half of a word, of what the planes before it left of an element.  Cut, not rounded, so that
// the largest f32 does not become infinite.  Single-pass products (two planes) of an infinity come out infinite, as from f32
// operands, if it meets the first plane of the other operand alone, whose second may be zero: the first plane has its sign, the
// second, which is left of it then, itself.
template <int PLANES>
__device__ __forceinline__ unsigned wide_part(float x, int plane) {
    const unsigned u = __float_as_uint(x);
    if (PLANES == 2 && plane == 0 && (u & 0x7fffffffu) == 0x7f800000u) return (u & 0x80000000u) | 0x3f800000u;
    return u & 0xffff0000u;
}

// Finishes the column sums.  And if the pass above found an operand that f16 does not hold: all of them again, as sums of three
// (or two) bf16, whose range is that of f32.  half_wide_exponent has their scale.
template <int PLANES>
__global__ void __launch_bounds__(kThreads)
split_wide_kernel(const __grid_constant__ ViewList list) {
    __shared__ float part[8][32];
    grid_dependency_trigger();
    grid_dependency_wait();
    unsigned status = 0;
    for (int i = threadIdx.x; i < list.statuses; i += kThreads) status |= __ldcg(list.status + i);
    const HalfColumns &sums = list.sums;
    if (sums.out) {
        const View &v = list.v[0];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per_strip = static_cast<int>(v.tiles_strip.d);
        for (int c32 = blockIdx.x * 32; c32 < v.cols; c32 += gridDim.x * 32) {
            // the blocks that took tiles of this strip
            const int strip = c32 / kTileCols, first = strip * per_strip, last = first + per_strip - 1;
            int b0 = static_cast<int>(static_cast<long long>(first) * list.statuses / list.tiles);
            while (b0 > 0 && first_tile_of(list, b0) > first) --b0;
            while (first_tile_of(list, b0 + 1) <= first) ++b0;
            int b1 = static_cast<int>(static_cast<long long>(last) * list.statuses / list.tiles);
            while (b1 > 0 && first_tile_of(list, b1) > last) --b1;
            while (first_tile_of(list, b1 + 1) <= last) ++b1;
            float s = 0.f;
            for (int b = b0 + warp; b <= b1; b += 8)
                s += __ldcg(sums.partial + static_cast<long long>(b + strip) * kTileCols + (c32 % kTileCols) + lane);
            part[warp][lane] = s;
            __syncthreads();
            if (warp == 0 && c32 + lane < v.cols) {
#pragma unroll
                for (int w = 1; w < 8; ++w) s += part[w][lane];
                sums.out[c32 + lane] = sums.accumulate ? sums.out[c32 + lane] + s : s;
            }
            __syncthreads();
        }
    }
    const bool unfit = __syncthreads_or(status & kUnfit), huge = __syncthreads_or(status & kHuge);
    if (blockIdx.x == 0 && threadIdx.x == 0) *list.verdict = (unfit ? kUnfit : 0u) | (huge ? kHuge : 0u);
    if (!unfit) return;
    for (int tile = blockIdx.x; tile < list.tiles; tile += gridDim.x) {
        int at = 0;
        while (at + 1 < list.count && tile >= list.v[at + 1].first_tile) ++at;
        const View &v = list.v[at];
        const Tile t = tile_at(v, tile - v.first_tile);
        const int c0 = t.c0 + (threadIdx.x & 63) * 8;
        const float scale = __uint_as_float(static_cast<unsigned>(127 + half_wide_exponent(__ldcg(v.exp), huge)) << 23);
        if (c0 >= v.pitch) continue;
        for (int r = t.r0 + (threadIdx.x >> 6); r < min(v.rows, t.r0 + kTileRows); r += 4) {
            const float *src = matrix_source(v, t.batch) + r * v.ld + c0;
            uint16_t *dst = v.dst + t.batch * v.matrix + static_cast<long long>(r) * v.pitch + c0;
            float x[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) x[c] = c0 + c < v.cols ? __ldg(src + c) * scale : 0.f;
#pragma unroll
            for (int plane = 0; plane < PLANES; ++plane) {
                uint4 out;
                unsigned *const o = &out.x;
#pragma unroll
                for (int c = 0; c < 8; c += 2) {
                    const unsigned a = wide_part<PLANES>(x[c], plane), b = wide_part<PLANES>(x[c + 1], plane);
                    o[c / 2] = (a >> 16) | b;
                    x[c] -= __uint_as_float(a);
                    x[c + 1] -= __uint_as_float(b);
                }
                *reinterpret_cast<uint4 *>(dst + plane * v.plane) = out;
            }
        }
    }
}

long long strips_of(const HalfView &v) { return (v.pitch + kTileCols - 1) / kTileCols; }
long long tiles_of(const HalfView &v) { return v.batch * ((v.rows + kTileRows - 1) / kTileRows) * strips_of(v); }

}  // namespace

size_t half_columns_bytes(const HalfView &first, int blocks) {
    return static_cast<size_t>(blocks + strips_of(first)) * kTileCols * sizeof(float);
}

int half_blocks(const HalfView *views, int count, int sm_count) {
    long long tiles = 0;
    for (int i = 0; i < count; ++i) tiles += tiles_of(views[i]);
    return static_cast<int>(std::min<long long>(tiles, static_cast<long long>(sm_count) * kBlocksPerSm));
}

int launch_split_half(const HalfView *views, int count, int planes, unsigned int *status, int blocks, const HalfColumns &sums,
                      cudaStream_t stream) {
    ViewList list{};
    list.count = count;
    list.status = status;
    list.statuses = blocks;
    list.verdict = status + blocks;
    list.sums = sums;
    long long tiles = 0;
    for (int i = 0; i < count; ++i) {
        const HalfView &h = views[i];
        View &v = list.v[i];
        v.src = h.src;
        v.dst = static_cast<uint16_t *>(h.dst);
        v.ld = h.ld;
        v.b0 = h.bstride[0]; v.b1 = h.bstride[1]; v.b2 = h.bstride[2];
        v.matrix = h.matrix;
        v.plane = h.plane;
        v.rows = static_cast<int>(h.rows);
        v.cols = static_cast<int>(h.cols);
        v.pitch = static_cast<int>(h.pitch);
        v.rows_d = make_fastdiv(h.rows);
        v.d1 = make_fastdiv(h.bshape[1]);
        v.d2 = make_fastdiv(h.bshape[2]);
        v.tiles_r = make_fastdiv((h.rows + kTileRows - 1) / kTileRows);
        v.tiles_strip = make_fastdiv(h.batch * ((h.rows + kTileRows - 1) / kTileRows));
        v.first_tile = static_cast<int>(tiles);
        v.total_rows = static_cast<unsigned>(h.batch * h.rows);
        v.vec = (reinterpret_cast<uintptr_t>(h.src) & 15) == 0 && h.ld % 4 == 0 && h.bstride[0] % 4 == 0 && h.bstride[1] % 4 == 0 &&
                h.bstride[2] % 4 == 0;
        v.exp = h.exp;
        tiles += tiles_of(h);
    }
    list.tiles = static_cast<int>(tiles);
    const dim3 grid(static_cast<unsigned>(blocks));
    const auto split = planes == 3 ? (sums.out ? split_half_kernel<true, true> : split_half_kernel<true, false>)
                                   : (sums.out ? split_half_kernel<false, true> : split_half_kernel<false, false>);
    cudaError_t e = launch_dependent(split, grid, dim3(kThreads), 0, stream, list);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "split_half_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("split_half_kernel");
    e = launch_dependent(planes == 3 ? split_wide_kernel<3> : split_wide_kernel<2>, grid, dim3(kThreads), 0, stream, list);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "split_wide_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("split_wide_kernel");
    return MNI_B200_OK;
}

}  // namespace mni
