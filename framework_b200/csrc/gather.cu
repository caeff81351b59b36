// Gathers of strided views into row-major buffers: contiguous(), permute_backward, and operands whose rows TMA cannot
// describe (a pitch that is not a multiple of 16 bytes).  HBM- or L2-bound: 8 bytes per element.
//
// The view's dimensions are first reduced on the host (extent-1 dimensions dropped, neighbours that are contiguous in
// source and destination merged); what is left picks the form of the copy.  Up to kMaxGathers views of a call go out
// as one launch.  Before, one form did everything with an element per thread and a 64-bit division per dimension:
// 27 us for a 12.6 MB head merge whose 25 MB of traffic take 4.
#include "internal.h"

#include <algorithm>

namespace mni {

namespace {

constexpr int kMaxDims = MNI_B200_MAX_DIMS;
constexpr int kThreads = 256;
// Units per thread of the row forms, all in flight together.  One up to 16 blocks per SM, where a second unit only takes
// warps away (4 MB head merge 4.5 us at four units, 3.2 at two, 2.6 at one); two beyond, where it covers the latency of
// the first (12.6 MB 6.2 / 4.9 / 5.0, 48x333x333 padded to 336 by 1.2 us faster at two than at four).
constexpr int kMaxItems = 2;
constexpr int kOneItemBlocksPerSm = 16;
constexpr int kTileU = 32, kTileI = 64;         // transposing form: source-contiguous x destination-contiguous

enum GatherKind {
    kRowsVec = 0,        // rows contiguous and aligned on both sides: a 16-byte unit each way
    kRowsQuad = 1,       // source rows contiguous, not aligned; destination padded to whole 16-byte units (pads become 0)
    kFlatQuad = 2,       // dense destination, any source: four consecutive elements per unit, which may cross rows
    kElements = 3,       // anything else, an element per unit
    kTranspose = 4,      // another dimension is the contiguous one of the source: tiles through shared memory
};

struct Gather {
    const float *src;
    float *dst;
    int kind, nd;                       // nd outer dimensions below
    FastDiv ext[kMaxDims];              // outer dimensions, outermost first
    long long sstr[kMaxDims];           // source strides of them
    long long dstr[kMaxDims];           // destination strides of them (transposing form)
    FastDiv units;                      // row forms: units per row; transposing form: tiles along the last dimension
    FastDiv tiles_u;                    // transposing form: tiles along the source-contiguous dimension
    int inner, eu;                      // extents of the last and of the source-contiguous dimension
    long long s_inner, d_u;             // source stride of the last dimension, destination stride of the other
    long long ld;                       // destination pitch of a row
    int items;                          // row forms: total units
    int elements;                       // kFlatQuad: total elements
    unsigned first;                     // first block of this gather
};
struct GatherList {
    Gather g[kMaxGathers];
    int count;
};

// Source address of the start of a row.
__device__ __forceinline__ const float *row_source(const Gather &g, int row) {
    const float *src = g.src;
    for (int d = g.nd - 1; d >= 0; --d) {
        const int q = fd_div(row, g.ext[d]);
        src += (row - q * static_cast<int>(g.ext[d].d)) * g.sstr[d];
        row = q;
    }
    return src;
}

// FLAT: some gather of the list is kFlatQuad, whose row crossings cost 8 registers a thread that the other forms keep for
// occupancy (12.6 MB head merge 6.1 us with them, 5.1 without).  Against an element per unit, four with one store take a
// permuted 500x333x65 from 48 us to 31.5.
template <int ITEMS, bool FLAT>
__global__ void __launch_bounds__(kThreads)
gather_kernel(const __grid_constant__ GatherList list) {
    __shared__ float tile[kTileI][kTileU + 1];
    grid_dependency_trigger();
    int j = 0;
    while (j + 1 < list.count && blockIdx.x >= list.g[j + 1].first) ++j;
    const Gather &g = list.g[j];
    const int block = static_cast<int>(blockIdx.x - g.first);
    grid_dependency_wait();
    if (g.kind == kTranspose) {
        const int rest = fd_div(block, g.units);
        const int i0 = (block - rest * static_cast<int>(g.units.d)) * kTileI;
        int rem = fd_div(rest, g.tiles_u);
        const int u0 = (rest - rem * static_cast<int>(g.tiles_u.d)) * kTileU;
        const float *src = g.src;
        float *dst = g.dst;
        for (int d = g.nd - 1; d >= 0; --d) {
            const int q = fd_div(rem, g.ext[d]);
            const int x = rem - q * static_cast<int>(g.ext[d].d);
            src += x * g.sstr[d];
            dst += x * g.dstr[d];
            rem = q;
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        float v[kTileI / 8];
#pragma unroll
        for (int k = 0; k < kTileI / 8; ++k) {
            const int i = i0 + warp + 8 * k;
            v[k] = (i < g.inner && u0 + lane < g.eu) ? __ldg(src + i * g.s_inner + u0 + lane) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < kTileI / 8; ++k) tile[warp + 8 * k][lane] = v[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTileU / 8; ++k) {
            const int u = u0 + warp + 8 * k;
            if (u >= g.eu) break;
#pragma unroll
            for (int h = 0; h < kTileI / 32; ++h) {
                const int i = i0 + lane + 32 * h;
                if (i < g.inner) dst[u * g.d_u + i] = tile[lane + 32 * h][warp + 8 * k];
            }
        }
        return;
    }
    const int base = block * (kThreads * ITEMS) + threadIdx.x;
    long long to[ITEMS];
    float4 v[ITEMS];
#pragma unroll
    for (int u = 0; u < ITEMS; ++u) {
        const int item = base + u * kThreads;
        if (item >= g.items) continue;
        if (FLAT && g.kind == kFlatQuad) {
            const int at = 4 * item;
            int row = fd_div(at, g.units), c = at - row * static_cast<int>(g.units.d);
            const float *src = row_source(g, row);
            to[u] = at;
            float e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (at + k >= g.elements) break;
                e[k] = __ldg(src + c * g.s_inner);
                if (++c == static_cast<int>(g.units.d) && k < 3 && at + k + 1 < g.elements) {
                    c = 0;
                    src = row_source(g, ++row);
                }
            }
            v[u] = make_float4(e[0], e[1], e[2], e[3]);
            continue;
        }
        const int row = fd_div(item, g.units), c = item - row * static_cast<int>(g.units.d);
        const float *src = row_source(g, row);
        to[u] = row * g.ld;
        if (g.kind == kElements) {
            to[u] += c;
            v[u].x = __ldg(src + c * g.s_inner);
        } else {
            to[u] += 4 * c;
            src += 4 * c;
            if (g.kind == kRowsVec) {
                v[u] = __ldg(reinterpret_cast<const float4 *>(src));
            } else {
                const int left = g.inner - 4 * c;
                v[u].x = __ldg(src);
                v[u].y = left > 1 ? __ldg(src + 1) : 0.f;
                v[u].z = left > 2 ? __ldg(src + 2) : 0.f;
                v[u].w = left > 3 ? __ldg(src + 3) : 0.f;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < ITEMS; ++u) {
        const int item = base + u * kThreads;
        if (item >= g.items) continue;
        if (g.kind == kElements) {
            g.dst[to[u]] = v[u].x;
        } else if (FLAT && g.kind == kFlatQuad && 4 * item + 4 > g.elements) {
            const float e[3] = {v[u].x, v[u].y, v[u].z};
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (4 * item + k < g.elements) g.dst[4 * item + k] = e[k];
        } else {
            *reinterpret_cast<float4 *>(g.dst + to[u]) = v[u];
        }
    }
}

// 64-bit form for views of 2^31 elements and more.
struct WideGather {
    int nd;
    long long shape[kMaxDims];
    long long stride[kMaxDims];
    long long ld_dst, total;
};
__global__ void __launch_bounds__(kThreads)
gather_wide_kernel(const float *__restrict__ src, float *__restrict__ dst, const WideGather a) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < a.total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        long long rem = i, off = 0;
        const long long last = a.shape[a.nd - 1];
        const long long c = rem % last;
        rem /= last;
        off += c * a.stride[a.nd - 1];
        const long long row = rem;
        for (int d = a.nd - 2; d >= 0; --d) {
            const long long q = rem % a.shape[d];
            rem /= a.shape[d];
            off += q * a.stride[d];
        }
        dst[row * a.ld_dst + c] = src[off];
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Fills `g` for one view; returns its tiles (transposing form, a block each) or units (the others).  The view has fewer
// than 2^31 elements, none of its extents is 0.
unsigned plan_gather(const GatherView &view, Gather &g) {
    const mni_b200_view &v = *view.src;
    // Dimensions outermost first: extent, source stride, destination stride.
    int64_t ext[kMaxDims + 1], ss[kMaxDims + 1], ds[kMaxDims + 1];
    int nd = 0;
    const int64_t inner_in = v.shape[v.ndim - 1];
    int64_t dstride[kMaxDims];
    dstride[v.ndim - 1] = 1;
    if (v.ndim > 1) dstride[v.ndim - 2] = view.ld_dst;
    for (int d = v.ndim - 3; d >= 0; --d) dstride[d] = dstride[d + 1] * v.shape[d + 1];
    for (int d = 0; d < v.ndim; ++d) {
        if (v.shape[d] == 1 && d != v.ndim - 1) continue;
        if (nd > 0 && ss[nd - 1] == v.stride[d] * v.shape[d] && ds[nd - 1] == dstride[d] * v.shape[d]) {
            ext[nd - 1] *= v.shape[d];
            ss[nd - 1] = v.stride[d];
            ds[nd - 1] = dstride[d];
        } else {
            ext[nd] = v.shape[d];
            ss[nd] = v.stride[d];
            ds[nd] = dstride[d];
            ++nd;
        }
    }
    const int last = nd - 1;
    const bool whole = ext[last] != inner_in;            // rows merged: the destination has no pads left
    const int64_t ld = whole ? ext[last] : view.ld_dst;
    g.src = v.ptr;
    g.dst = view.dst;
    g.inner = static_cast<int>(ext[last]);
    g.s_inner = ss[last];
    g.ld = ld;
    // A source-contiguous dimension other than the last, wide enough on both sides for tiles.
    int u = -1;
    if (ss[last] != 1)
        for (int d = 0; d < last; ++d)
            if (ss[d] == 1 && ext[d] >= 8 && (u < 0 || ext[d] > ext[u])) u = d;
    if (u >= 0 && ext[last] >= 8) {
        g.kind = kTranspose;
        g.eu = static_cast<int>(ext[u]);
        g.d_u = ds[u];
        g.nd = 0;
        int64_t others = 1;
        for (int d = 0; d < last; ++d) {
            if (d == u) continue;
            g.ext[g.nd] = make_fastdiv(ext[d]);
            g.sstr[g.nd] = ss[d];
            g.dstr[g.nd] = ds[d];
            ++g.nd;
            others *= ext[d];
        }
        const int64_t ti = (ext[last] + kTileI - 1) / kTileI, tu = (ext[u] + kTileU - 1) / kTileU;
        g.units = make_fastdiv(ti);
        g.tiles_u = make_fastdiv(tu);
        g.items = 0;
        return static_cast<unsigned>(others * ti * tu);
    }
    int64_t rows = 1;
    bool aligned = aligned16(v.ptr);
    g.nd = last;
    for (int d = 0; d < last; ++d) {
        g.ext[d] = make_fastdiv(ext[d]);
        g.sstr[d] = ss[d];
        rows *= ext[d];
        aligned = aligned && ss[d] % 4 == 0;
    }
    const bool units4 = (ss[last] == 1 || ext[last] == 1) && aligned16(view.dst) && (rows == 1 || ld % 4 == 0);
    if (units4 && aligned && ext[last] % 4 == 0) g.kind = kRowsVec;
    else if (units4 && (rows == 1 ? ext[last] % 4 == 0 : ld - ext[last] < 4 && ld != ext[last])) g.kind = kRowsQuad;
    else if (aligned16(view.dst) && (rows == 1 || ld == ext[last])) g.kind = kFlatQuad;
    else g.kind = kElements;
    g.elements = static_cast<int>(rows * ext[last]);
    const int64_t units = g.kind == kElements || g.kind == kFlatQuad ? ext[last] : (ext[last] + 3) / 4;
    g.units = make_fastdiv(units);
    g.items = static_cast<int>(g.kind == kFlatQuad ? (rows * ext[last] + 3) / 4 : rows * units);
    return static_cast<unsigned>(g.items);
}

}  // namespace

int launch_gather(const GatherView *views, int count, cudaStream_t stream) {
    GatherList list;
    list.count = 0;
    unsigned sizes[kMaxGathers];
    long long units = 0;
    bool flat = false;
    for (int i = 0; i < count; ++i) {
        const mni_b200_view &v = *views[i].src;
        long long total = 1;
        for (int d = 0; d < v.ndim; ++d) total *= v.shape[d];
        if (total == 0) continue;
        if (total >= (1LL << 31) - 4 * kThreads * kMaxItems || views[i].ld_dst >= (1LL << 31)) {
            WideGather a{};
            a.nd = v.ndim;
            for (int d = 0; d < v.ndim; ++d) { a.shape[d] = v.shape[d]; a.stride[d] = v.stride[d]; }
            a.ld_dst = views[i].ld_dst;
            a.total = total;
            const long long want = (total + kThreads - 1) / kThreads;
            gather_wide_kernel<<<static_cast<unsigned>(std::min<long long>(want, device_sm_count() * 16LL)), kThreads, 0, stream>>>(
                v.ptr, views[i].dst, a);
            MNI_LAUNCH_CHECK("gather_wide_kernel");
            continue;
        }
        sizes[list.count] = plan_gather(views[i], list.g[list.count]);
        if (list.g[list.count].kind != kTranspose) units += sizes[list.count];
        if (list.g[list.count].kind == kFlatQuad) flat = true;
        ++list.count;
    }
    const bool one = units <= static_cast<long long>(device_sm_count()) * kOneItemBlocksPerSm * kThreads;
    const unsigned per_block = kThreads * (one ? 1 : kMaxItems);
    unsigned blocks = 0;
    for (int i = 0; i < list.count; ++i) {
        list.g[i].first = blocks;
        blocks += list.g[i].kind == kTranspose ? sizes[i] : (sizes[i] + per_block - 1) / per_block;
    }
    if (blocks == 0) return MNI_B200_OK;
    const auto kernel = one ? (flat ? gather_kernel<1, true> : gather_kernel<1, false>)
                            : (flat ? gather_kernel<kMaxItems, true> : gather_kernel<kMaxItems, false>);
    const cudaError_t e = launch_dependent(kernel, dim3(blocks), dim3(kThreads), 0, stream, list);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "gather_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("gather_kernel");
    return MNI_B200_OK;
}

}  // namespace mni
