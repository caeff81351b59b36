// C ABI of libmni_b200.so: argument checking, view classification, path selection and
// scratch management.  All arithmetic happens in the kernels of gemm_tcgen05.cu,
// skinny.cu and pointwise.cu; there is no host or library (cuBLAS) fallback.
#include "internal.h"

#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

namespace mni {

std::atomic<uint64_t> g_launches{0};

namespace {

thread_local char t_error[512] = "";

__device__ unsigned int g_err_word;   // first timeout code recorded by any kernel of the library

constexpr int kMaxDevices = 64;

struct DeviceState {
    std::mutex mu;
    bool init = false;
    int sm_count = 0;
    int sm_reserve = 0;           // SMs the tensor-core launches leave free (mni_b200_sm_reserve)
    int cc_major = 0;
    uint8_t *ws = nullptr;        // library-owned scratch
    size_t ws_bytes = 0;
    bool ws_recorded = false;     // some graph holds its address
    size_t refused = SIZE_MAX;    // the least that could not be had for 16-bit planes, and what was free then: not tried again
    size_t refused_free = 0;      // until more is (or mni_b200_release)
    std::vector<uint8_t *> retired;   // scratch outgrown since, kept for the graphs that hold its address (mni_b200_release frees it)
    uint8_t *user_ws = nullptr;   // caller-provided scratch (takes precedence)
    size_t user_bytes = 0;
    unsigned int *err_word = nullptr;
    // Second stream of small backward calls: dA and dB of a small problem each occupy a fraction of
    // the GPU, so they are issued side by side (fork / join through events; also under stream capture).
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};
DeviceState g_dev[kMaxDevices];

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// x^n in f32 the way Rust's f32::powi evaluates it (ops/optimizer.rs:26-27 call it for the bias corrections):
// binary exponentiation from the lowest exponent bit up -- multiply the result in when the bit is set,
// square the base between bits -- every product rounded to f32.  O(log n) and, from n = 4 on, rounded
// differently from n successive multiplications.
float powi_f32(float x, uint32_t n) {
    float r = 1.0f;
    while (true) {
        if (n & 1u) r *= x;
        n >>= 1;
        if (n == 0) break;
        x *= x;
    }
    return r;
}

// Largest M*N*K*batch for which the two gradient products of a backward call are issued side by side.
double overlap_work_limit() {
    const char *v = env_value("MNI_B200_BWD_OVERLAP_WORK");
    return v ? atof(v) : 4.0e9;   // measured: helps up to the attention-shaped products (1.6e9), neutral beyond
}

// Row counts up to which the streaming kernels beat the tensor path (measured at K = N = 4096 with a weight
// that is not in L2: dx 19.4 vs 23.6 us at 5 rows and 31.0 vs 23.7 at 8; dW 14 vs 16.9 at 8 rows, 15.5 at 12, 20.7 at
// 15: beyond 8 rows it goes with the calls of few rows below).  The forward's limit depends on which of its two kernels can
// run: skinny_fwd_row_limit.
constexpr int64_t kSkinnyDxRows = 5, kSkinnyDwRows = 8;

// Rows up to which the warp-level streaming kernels (rows.cu) take a product the FFMA kernels above do not.  From 16
// rows, the narrowest tile of the tensor path, that path wastes nothing on an aligned weight; one whose rows are not
// 16-byte aligned it would have to gather first.
constexpr int64_t kRowsAligned = 15, kRowsUnaligned = 16;
// ... of an aligned weight with short contractions only, or up to 16 M elements with at least as many outputs: larger ones the
// tensor path streams better (9 rows, weight not in L2, us here / there: 1024 x 4096 forward 7.9 / 10.4, 4096 x 4096 19.1 / 19.2,
// 2792 x 3880 14.6 / 15.7 and its dx 19.9 / 15.6, 8192 x 8192 66 / 57, 4096 x 12000 75 / 55, 6000 x 3000 27 / 21).
constexpr int64_t kRowsShort = 1024, kRowsElements = 1 << 24;

// Limits of the one-launch f32 kernel (tiny.cu): it needs about 1.9 us and 1 us per 64 contraction elements, up to M * N * K =
// 8 M (192^3: forward 5.0 us against 7.7, backward 5.8 against 8.9; 256^3 is level; K = 512 loses), and up to so many 32 x 32
// tiles of output -- three a block slot and more queue up and store element by element (2048 x 1 x 4096, 8192 tiles: 62 us
// against 13).  An eager call gains from one launch in place of two to four (491 x 8 x 1746, 880 tiles: 8.5 against 11.5), the
// two gradients of a backward call more (13 x 5616 x 99, 880 tiles: 11.0 against 15.6; 48 x 18120 x 3, 1701: 16.7 / 17.1).  Under
// capture only device time counts, and one product with aligned output rows and more than the 64 rows that are computed exchanged
// is the tensor path's from fewer tiles on (104 x 1 x 4776, 600 tiles: 7.0 against 5.5; but 20 x 3 x 16904 5.7 / 7.2).
constexpr int64_t kTinyContraction = 320, kTinyContractionFewRows = 128;
constexpr int kTinyWork = 1 << 23;
constexpr int64_t kTinyTiles = 900, kTinyTilesBoth = 1200, kTinyTilesCaptured = 400;
// Up to 8 rows the streaming kernels are the competition.  For one product they win but where the tiles are few and five rows
// or more, or a short contraction, share them (8 x 8 x 4512 forward 3.3 us against 4.8, 8 x 90 x 1656 4.1 / 6.3; but 8 x 128 x
// 8192 6.1 / 4.8, 1 x 128 x 4096 5.6 / 3.1, input gradient 8 x 496 x 8 2.7 / 2.6).  A backward call for both gradients they make in two launches on two
// streams: eager 8 x 12704 x 8 8.1 us against 14.8, captured 7.7 / 6.3, 4 x 4096 x 64 5.7 / 3.8, 8 x 2048 x 127 5.5 / 6.7.
constexpr int64_t kTinyTilesFewRows = 256, kTinyTilesFewest = 8;

bool env_flag(const char *name, int dflt) { return env_int(name, dflt) != 0; }

// Bump allocator over the device's scratch.  In dry mode nothing is touched: the
// same host logic runs and only the byte count is produced (workspace_query).
struct Arena {
    DeviceState *st = nullptr;
    bool dry = false;
    size_t used = 0;
    std::vector<std::pair<size_t, size_t>> blocks;   // (offset, bytes) in request order
    size_t reserve(size_t bytes) {
        const size_t off = used;
        used += (bytes + 255) & ~static_cast<size_t>(255);
        return off;
    }
};

int device_state(DeviceState **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_DEVICE, "no CUDA device: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(MNI_B200_ERR_DEVICE, "device ordinal %d out of range", dev);
    DeviceState &st = g_dev[dev];
    // First use of a device: under the device's lock, so that two host threads that make their first
    // call together initialise it once (init is only ever read or written with the lock held).
    std::lock_guard<std::mutex> lock(st.mu);
    if (!st.init) {
        cudaDeviceProp prop;
        e = cudaGetDeviceProperties(&prop, dev);
        if (e != cudaSuccess) return fail(MNI_B200_ERR_DEVICE, "cudaGetDeviceProperties: %s", cudaGetErrorString(e));
        if (prop.major != 10)
            return fail(MNI_B200_ERR_DEVICE,
                        "device %d is compute capability %d.%d; this library only carries sm_100a code", dev,
                        prop.major, prop.minor);
        st.sm_count = prop.multiProcessorCount;
        st.cc_major = prop.major;
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_err_word);
        if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        st.err_word = static_cast<unsigned int *>(p);
        e = cudaMemset(st.err_word, 0, sizeof(unsigned int));
        if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "cudaMemset: %s", cudaGetErrorString(e));
        if (!st.side) e = cudaStreamCreateWithFlags(&st.side, cudaStreamNonBlocking);
        if (e == cudaSuccess && !st.ev_fork) e = cudaEventCreateWithFlags(&st.ev_fork, cudaEventDisableTiming);
        if (e == cudaSuccess && !st.ev_join) e = cudaEventCreateWithFlags(&st.ev_join, cudaEventDisableTiming);
        if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "side stream set-up: %s", cudaGetErrorString(e));
        st.init = true;
    }
    *out = &st;
    return MNI_B200_OK;
}

// True while `stream` records into a CUDA graph.
bool stream_is_capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
        cudaGetLastError();   // the legacy stream beside another stream's capture: not capturing itself
        return false;
    }
    return status != cudaStreamCaptureStatusNone;
}

// What is allocated where `bytes` of scratch are needed.
size_t scratch_for(size_t bytes) { return bytes + bytes / 4 + (1u << 20); }

// Whether scratch of this size, or less, was refused and there is no more memory than then.  Growing frees and allocates, which
// calls that go on without it must not do each time.
bool scratch_refused(const DeviceState &st, size_t bytes) {
    if (bytes < st.refused) return false;
    size_t free = 0, total = 0;
    if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return free <= st.refused_free || free + (st.ws_recorded ? 0 : st.ws_bytes) < scratch_for(bytes);
}
void note_refused(DeviceState &st, size_t bytes) {
    size_t free = 0, total = 0;
    if (cudaMemGetInfo(&free, &total) != cudaSuccess) cudaGetLastError();
    st.refused = bytes;
    st.refused_free = free;
}

// Makes `bytes` of scratch available and returns its base.
int scratch_base(DeviceState &st, size_t bytes, cudaStream_t stream, uint8_t **base) {
    if (st.user_ws) {
        if (bytes > st.user_bytes)
            return fail(MNI_B200_ERR_WORKSPACE, "caller-provided scratch holds %zu bytes, %zu needed", st.user_bytes,
                        bytes);
        *base = st.user_ws;
        return MNI_B200_OK;
    }
    if (bytes > st.ws_bytes) {
        const size_t want = scratch_for(bytes);
        // Growing frees the old buffer, which a capturing stream must not do (it would end the capture in
        // an error).
        if (st.ws && stream_is_capturing(stream))
            return fail(MNI_B200_ERR_WORKSPACE,
                        "scratch would have to grow from %zu to %zu bytes while the stream is capturing: run the call "
                        "once before the capture, or hand the library a buffer (mni_b200_workspace_set)",
                        st.ws_bytes, bytes);
        // What there is stays if the larger buffer cannot be had: calls that fit in it may be captured later on.
        const bool keep = st.ws && st.ws_recorded;
        const size_t old_bytes = keep ? 0 : st.ws_bytes;
        if (st.ws && !keep) {
            // cudaFree waits for work that may still read the old buffer.
            cudaError_t e = cudaFree(st.ws);
            st.ws = nullptr;
            st.ws_bytes = 0;
            if (e != cudaSuccess) return fail(MNI_B200_ERR_WORKSPACE, "cudaFree(scratch): %s", cudaGetErrorString(e));
        }
        void *p = nullptr;
        const cudaError_t e = cudaMalloc(&p, want);
        if (e != cudaSuccess) {
            cudaGetLastError();
            if (old_bytes && cudaMalloc(&p, old_bytes) == cudaSuccess) {
                st.ws = static_cast<uint8_t *>(p);
                st.ws_bytes = old_bytes;
            }
            cudaGetLastError();
            return fail(MNI_B200_ERR_WORKSPACE, "cudaMalloc(%zu) for scratch failed: %s", want, cudaGetErrorString(e));
        }
        if (keep) st.retired.push_back(st.ws);
        st.ws_recorded = false;
        st.ws = static_cast<uint8_t *>(p);
        st.ws_bytes = want;
    }
    if (!st.ws_recorded && stream_is_capturing(stream)) st.ws_recorded = true;
    *base = st.ws;
    return MNI_B200_OK;
}

// Where a kernel leaves a number for the host: slots of pinned memory, one per call that is waiting.  The pool is
// process-wide (portable pinned memory), bounded, and a slot goes back when its call returns.
struct NormSlotLease {
    NormSlot *slot = nullptr;
    unsigned seq = 0;
    static constexpr int kSlots = 64;
    struct Pool {
        std::mutex mu;
        NormSlot *base = nullptr;
        uint64_t used = 0;         // bit per slot
        unsigned next_seq = 0;
    };
    static Pool &pool() { static Pool p; return p; }
    int take() {
        Pool &p = pool();
        std::unique_lock<std::mutex> lock(p.mu);
        if (!p.base) {
            void *m = nullptr;
            const cudaError_t e = cudaHostAlloc(&m, kSlots * sizeof(NormSlot), cudaHostAllocPortable | cudaHostAllocMapped);
            if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "cudaHostAlloc: %s", cudaGetErrorString(e));
            memset(m, 0, kSlots * sizeof(NormSlot));
            p.base = static_cast<NormSlot *>(m);
        }
        while (~p.used == 0) {                // every slot is out: some call returns its own soon
            lock.unlock();
            std::this_thread::yield();
            lock.lock();
        }
        const int i = __builtin_ctzll(~p.used);
        p.used |= 1ull << i;
        slot = p.base + i;
        if (++p.next_seq == 0) ++p.next_seq;
        seq = p.next_seq;
        return MNI_B200_OK;
    }
    // Waits until the kernel has written the slot, or until the stream has ended without doing so.
    int wait(cudaStream_t stream) {
        volatile unsigned *const arrived = &slot->seq;
        for (uint64_t spins = 1; *arrived != seq; ++spins) {
            if ((spins & 0x3fff) != 0) continue;
            const cudaError_t e = cudaStreamQuery(stream);
            if (e == cudaErrorNotReady) continue;
            if (e == cudaSuccess && *arrived == seq) break;
            return fail(MNI_B200_ERR_CUDA, "the norm did not arrive: %s", cudaGetErrorString(e));
        }
        std::atomic_thread_fence(std::memory_order_acquire);
        return MNI_B200_OK;
    }
    ~NormSlotLease() {
        if (!slot) return;
        Pool &p = pool();
        std::lock_guard<std::mutex> lock(p.mu);
        p.used &= ~(1ull << (slot - p.base));
    }
};

// ------------------------------------------------------------------ shapes
int64_t prod(const int64_t *s, int n) {
    int64_t p = 1;
    for (int i = 0; i < n; ++i) p *= s[i];
    return p;
}

// utils.rs:3-20
int broadcast_shape(const int64_t *a, int an, const int64_t *b, int bn, int64_t *out) {
    const int nd = std::max(an, bn);
    for (int i = 0; i < nd; ++i) {
        const int64_t da = i < nd - an ? 1 : a[i - (nd - an)];
        const int64_t db = i < nd - bn ? 1 : b[i - (nd - bn)];
        if (da == db) out[i] = da;
        else if (da == 1) out[i] = db;
        else if (db == 1) out[i] = da;
        else return -1;
    }
    return nd;
}

int check_view(const mni_b200_view *v, const char *name, int min_nd) {
    if (!v) return fail(MNI_B200_ERR_ARG, "%s is null", name);
    if (v->ndim < min_nd) return fail(MNI_B200_ERR_NDIM, "matmul requires at least 2D tensors (%s has %d)", name, v->ndim);
    if (v->ndim > MNI_B200_MAX_DIMS) return fail(MNI_B200_ERR_ARG, "%s has %d dims (max %d)", name, v->ndim, MNI_B200_MAX_DIMS);
    for (int d = 0; d < v->ndim; ++d) {
        if (v->shape[d] < 0 || v->stride[d] < 0) return fail(MNI_B200_ERR_ARG, "%s has a negative extent or stride", name);
        if (v->shape[d] > 0x7fffffffLL) return fail(MNI_B200_ERR_TOO_LARGE, "%s dim %d = %lld exceeds 2^31-1", name, d, (long long)v->shape[d]);
    }
    if (!v->ptr && prod(v->shape, v->ndim) > 0) return fail(MNI_B200_ERR_ARG, "%s has a null data pointer", name);
    return MNI_B200_OK;
}

// A matrix operand read through a TMA descriptor.  `transposed` selects which of the
// view's last two dims is the contraction dim: false -> [.., rows, k], true -> [.., k, rows].
// Returns false if the view cannot be described (then the caller packs it first).
bool view_to_operand(const mni_b200_view &v, bool transposed, Operand &op) {
    const int nd = v.ndim;
    const int64_t s_r = transposed ? v.stride[nd - 1] : v.stride[nd - 2];
    const int64_t s_k = transposed ? v.stride[nd - 2] : v.stride[nd - 1];
    op.ptr = v.ptr;
    op.rows = transposed ? v.shape[nd - 1] : v.shape[nd - 2];
    op.kdim = transposed ? v.shape[nd - 2] : v.shape[nd - 1];
    if ((reinterpret_cast<uintptr_t>(v.ptr) & 15) != 0) return false;
    const bool k_ok = (s_k == 1 || op.kdim == 1) && (op.rows == 1 || (s_r > 0 && s_r % 4 == 0));
    const bool mn_ok = (s_r == 1 || op.rows == 1) && (op.kdim == 1 || (s_k > 0 && s_k % 4 == 0));
    if (k_ok) {
        op.k_major = true;
        op.ld = s_r;
    } else if (mn_ok) {
        op.k_major = false;
        op.ld = s_k;
    } else {
        return false;
    }
    // Batch dims: drop extent-1 dims, merge dims that are contiguous with each other.
    int64_t bs[MNI_B200_MAX_DIMS], bt[MNI_B200_MAX_DIMS];
    int nb = 0;
    op.batch = 1;
    for (int d = 0; d < nd - 2; ++d) {
        op.batch *= v.shape[d];
        if (v.shape[d] == 1) continue;
        if (nb > 0 && bt[nb - 1] == v.stride[d] * v.shape[d]) {
            bs[nb - 1] *= v.shape[d];
            bt[nb - 1] = v.stride[d];
        } else {
            bs[nb] = v.shape[d];
            bt[nb] = v.stride[d];
            ++nb;
        }
    }
    if (nb > 3) return false;
    for (int i = 0; i < 3; ++i) { op.bshape[i] = 1; op.bstride[i] = 0; }
    for (int i = 0; i < nb; ++i) {
        if (bt[i] <= 0 || bt[i] % 4 != 0) return false;
        if (bs[i] > 0x7fffffffLL) return false;
        op.bshape[3 - nb + i] = bs[i];
        op.bstride[3 - nb + i] = bt[i];
    }
    return true;
}

struct Call {
    DeviceState *st;
    Arena arena;
    cudaStream_t stream;
    uint32_t flags;
    uint8_t *base = nullptr;   // resolved scratch base (real mode, second pass)
    bool capturing = false;    // the stream records into a graph
    int flag_bank = 0;         // 1 while launches go to the library's side stream / for the second product of a pair
    int dep_mode = 0;          // GemmProblem::dep_mode of the tensor-path launches issued now
    bool used_half = false;    // some product of the call is computed from 16-bit halves
    bool no_half = false;      // there is no scratch for operands as 16-bit halves
    GemmFinish *defer = nullptr;       // where the next product leaves its split-K finish instead of launching it
    int sm_share = 1;          // 2 while grad_a and grad_b run side by side: each is planned for half of the SMs
    std::string *plan_log = nullptr;   // mni_b200_plan_describe: one line per launch the call would make
    const char *label = "";            // which product the launches logged now belong to
    void note(const std::string &what) const {
        if (plan_log) *plan_log += std::string(label) + what + "\n";
    }
    // SMs the persistent tensor-core grids are planned for: all of them minus the caller's reservation, divided
    // between the products that run at the same time (kept even, CTA pairs take two)
    int gemm_sms(int share) const { return std::max(8, ((st->sm_count - st->sm_reserve) / share) & ~1); }
    int gemm_sms() const { return gemm_sms(sm_share); }
    bool dry() const { return arena.dry; }
    float *at(size_t off) const { return reinterpret_cast<float *>(base + off); }
};

// Gathers views into scratch as [batch_flat, R, C] with the last dim padded to a multiple of 4, all in one launch.
// Each *use[i] is replaced by the view of its packed copy, which `packed[i]` holds.
int pack_views(Call &c, const mni_b200_view **const *use, mni_b200_view *packed, int count) {
    GatherView jobs[kMaxGathers];
    for (int i = 0; i < count; ++i) {
        const mni_b200_view &v = **use[i];
        const int nd = v.ndim;
        const int64_t cols = v.shape[nd - 1], rows = v.shape[nd - 2];
        const int64_t ld = std::max<int64_t>(4, round_up(cols, 4));
        const int64_t batch = prod(v.shape, nd - 2);
        const size_t off = c.arena.reserve(static_cast<size_t>(batch * rows * ld) * sizeof(float));
        mni_b200_view &q = packed[i];
        q.ndim = 3;
        q.shape[0] = batch; q.shape[1] = rows; q.shape[2] = cols;
        q.stride[0] = rows * ld; q.stride[1] = ld; q.stride[2] = 1;
        q.ptr = c.dry() ? reinterpret_cast<const float *>(static_cast<uintptr_t>(256)) : c.at(off);
        jobs[i] = GatherView{&v, c.dry() ? nullptr : c.at(off), ld};
        c.note("gather of a strided operand into scratch");
    }
    int rc = MNI_B200_OK;
    if (!c.dry()) rc = launch_gather(jobs, count, c.stream);
    for (int i = 0; i < count; ++i) *use[i] = &packed[i];
    return rc;
}

// The operands TMA cannot describe (or all of them, under the test flag) are gathered first.  A gathered operand serves
// every product of the call, whichever of its two matrix dims is contracted: the copy is describable either way.
int pack_undescribable(Call &c, std::initializer_list<const mni_b200_view **> uses, mni_b200_view *packed) {
    const mni_b200_view **need[kMaxGathers];
    int count = 0;
    for (const mni_b200_view **u : uses) {
        Operand probe;
        if ((c.flags & MNI_B200_FORCE_PACK) != 0 || !view_to_operand(**u, false, probe)) need[count++] = u;
    }
    return count ? pack_views(c, need, packed, count) : static_cast<int>(MNI_B200_OK);
}

int make_operand(const mni_b200_view &v, bool transposed, Operand &op) {
    return view_to_operand(v, transposed, op) ? static_cast<int>(MNI_B200_OK)
                                              : fail(MNI_B200_ERR_ARG, "operand is not describable");
}

int run_gemm(Call &c, GemmProblem &p) {
    p.fast_tf32 = (c.flags & MNI_B200_PRECISION_TF32) != 0;
    p.force_splits = static_cast<int>((c.flags >> 16) & 0xffu);
    p.flag_bank = c.flag_bank;
    p.dep_mode = c.dep_mode;
    p.beside = c.sm_share > 1;
    if (p.M > 0x7fffffffLL || p.N > 0x7fffffffLL || p.K > 0x7fffffffLL || p.batch * p.fold > 0x7fffffffLL ||
        p.batch * ((p.M + 127) / 128) * ((p.N + 63) / 64) > 0x3fffffffLL)
        return fail(MNI_B200_ERR_TOO_LARGE, "GEMM %lld x %lld x %lld (batch %lld) exceeds the kernels' int32 indexing",
                    (long long)p.M, (long long)p.N, (long long)p.K, (long long)p.batch);
    const size_t pbytes = gemm_tc_partial_bytes(p, c.gemm_sms());
    size_t poff = 0;
    if (pbytes) poff = c.arena.reserve(pbytes);
    if (c.plan_log) c.note(gemm_tc_describe(p, c.gemm_sms()));
    if (c.dry()) return MNI_B200_OK;
    return launch_gemm_tc(p, pbytes ? c.at(poff) : nullptr, c.st->err_word, c.gemm_sms(), c.stream, c.defer);
}

// ------------------------------------------------------------------ large products from 16-bit halves
// A view as matrices with a unit stride along their columns (swapped: the view's last two dims are exchanged for that).
bool view_to_half(const mni_b200_view &v, HalfView &h, bool *swapped) {
    const int nd = v.ndim;
    *swapped = v.stride[nd - 1] != 1;
    if (*swapped && v.stride[nd - 2] != 1) return false;
    const int r = *swapped ? nd - 1 : nd - 2, k = *swapped ? nd - 2 : nd - 1;
    h.src = v.ptr;
    h.rows = v.shape[r];
    h.cols = v.shape[k];
    h.ld = v.stride[r];
    int nb = 0;
    int64_t bs[MNI_B200_MAX_DIMS], bt[MNI_B200_MAX_DIMS];
    h.batch = 1;
    for (int d = 0; d < nd - 2; ++d) {
        h.batch *= v.shape[d];
        if (v.shape[d] == 1) continue;
        if (v.stride[d] == 0) return false;
        if (nb > 0 && bt[nb - 1] == v.stride[d] * v.shape[d]) {
            bs[nb - 1] *= v.shape[d];
            bt[nb - 1] = v.stride[d];
        } else {
            bs[nb] = v.shape[d];
            bt[nb] = v.stride[d];
            ++nb;
        }
    }
    if (nb > 3) return false;
    for (int i = 0; i < 3; ++i) { h.bshape[i] = 1; h.bstride[i] = 0; }
    for (int i = 0; i < nb; ++i) { h.bshape[3 - nb + i] = bs[i]; h.bstride[3 - nb + i] = bt[i]; }
    h.pitch = round_up(h.cols, 64);
    h.matrix = h.rows * h.pitch;
    h.plane = h.batch * h.matrix;
    return h.ld >= 0 && h.batch * h.rows < 0x7fffffffLL && h.batch * ((h.rows + 15) / 16) * ((h.pitch + 511) / 512) < 0x1fffffffLL;
}

// The 16-bit planes of a call's operands.
struct Halves {
    HalfView view[kMaxHalves];
    bool swapped[kMaxHalves];
    int count = 0, blocks = 0, planes = 3;
    unsigned int *status = nullptr;
    // operand i with its last dim contracted, or (transposed) the one before
    HalfOperand operand(int i, bool transposed) const {
        const HalfView &v = view[i];
        HalfOperand o;
        o.ptr = v.dst;
        o.k_major = swapped[i] == transposed;
        o.rows = o.k_major ? v.rows : v.cols;
        o.kdim = o.k_major ? v.cols : v.rows;
        o.pitch = v.pitch; o.matrix = v.matrix; o.plane = v.plane;
        o.batch = v.batch;
        o.planes = planes;
        o.exp = v.exp;
        return o;
    }
};

// Whether a call may be computed from 16-bit planes, and is large enough for it to be worth finding out whether that pays.  Below
// the line it seldom does; f32 operands / planes, us: forward 1280^3 30 / 38, 1024 x 768 x 3072 32 / 34, 1536^3 38 / 45; backward
// 1280^3 46 / 47, 1024 x 3072 x 768 43 / 57, 8192 x 256 x 1024 44 / 62, but 1536^3 64 / 56 and 1000 x 1333 x 2777 113 / 89.
constexpr double kHalfWork = 4.0e9;                // M * N * K of its products
bool half_possible(const Call &c, double work) {
    const uint32_t forced = MNI_B200_FORCE_TENSOR_PATH | MNI_B200_FORCE_SKINNY_PATH | MNI_B200_FORCE_PACK;
    return !c.no_half && (c.flags & forced) == 0 && ((c.flags >> 16) & 0xffu) == 0 &&
           (work >= kHalfWork || env_int("MNI_B200_HALF", -1) > 0);
}
// Whether it pays: `f32_us` the estimate for the products from f32 operands, `half_us` from 16-bit planes, which the pass over the
// operands' `elements` comes on top of (8 bytes an element, 6 in single-pass mode, at 5.2 TB/s, and 7 us for its two launches).
// Measured with f32 operands / 16-bit planes, us, in a loop: forward 2048 x 768 x 3072 56 / 63, 2048^3 67 / 68, 8192 x 768 x 3072
// 142 / 131, 4096 x 1024 x 4096 133 / 110, 4096^3 516 / 339, 1024 x 8192 x 1024 70 / 83, 8192 x 8192 x 512 252 / 282; backward
// 2048 x 768 x 3072 113 / 107, 2048^3 133 / 107, 8192 x 768 x 3072 322 / 242, 4096^3 1071 / 612, 512 x 4096 x 4096 144 / 147;
// single pass forward 3072^3 79 / 80, 4096^3 219 / 159, backward 162 / 128, 440 / 258.  Near the line, with three sets of operands
// in turn: backward 2048 x 1024 x 2048 77 / 69, 2048^2 x 1024 78 / 74, 2048 x 3072 x 768 88 / 84, 4096 x 512 x 2048 82 / 77, 3000 x
// 700 x 2000 96 / 79, 1500 x 1024 x 4096 118 / 96.  That is at the clocks the power cap leaves; in the first 2 ms after a pause
// the same six take 66 / 68, 67 / 74, 74 / 85, 70 / 77, 84 / 78, 101 / 92.  MNI_B200_HALF=0 / 1: never / wherever it can be done.
bool half_pays(const Call &c, double f32_us, double half_us, double elements) {
    const int env = env_int("MNI_B200_HALF", -1);
    if (env >= 0) return env > 0;
    const bool single = (c.flags & MNI_B200_PRECISION_TF32) != 0;
    return half_us + 7.0 + (single ? 6.0 : 8.0) * elements / 5.2e6 < (single ? 0.92 : 0.96) * f32_us;
}
// Gathering an operand that TMA cannot describe, in microseconds.
double gather_us(const mni_b200_view &v) {
    Operand probe;
    return view_to_operand(v, false, probe) ? 0.0 : 3.0 + 8.0 * static_cast<double>(prod(v.shape, v.ndim)) / 4.0e6;
}

// sums_out: also the column sums of the first view.
int make_halves(Call &c, std::initializer_list<const mni_b200_view *> views, Halves &h, float *sums_out = nullptr, bool accumulate = false) {
    for (const mni_b200_view *v : views) {
        if (!view_to_half(*v, h.view[h.count], &h.swapped[h.count])) return fail(MNI_B200_ERR_ARG, "internal: operand has no halves");
        ++h.count;
    }
    h.planes = (c.flags & MNI_B200_PRECISION_TF32) != 0 ? 2 : 3;
    h.blocks = half_blocks(h.view, h.count, c.st->sm_count);
    const size_t words = static_cast<size_t>(h.blocks) + 1 + kMaxHalves, head = c.arena.reserve(4 * words);
    size_t at[kMaxHalves];
    for (int i = 0; i < h.count; ++i) at[i] = c.arena.reserve(static_cast<size_t>(h.view[i].plane) * 2 * h.planes);
    const size_t sums_at = sums_out ? c.arena.reserve(half_columns_bytes(h.view[0], h.blocks)) : 0;
    c.used_half = true;
    c.note("operands into 16-bit planes");
    if (c.dry()) return MNI_B200_OK;
    h.status = reinterpret_cast<unsigned int *>(c.at(head));
    for (int i = 0; i < h.count; ++i) {
        h.view[i].dst = c.at(at[i]);
        h.view[i].exp = reinterpret_cast<int *>(h.status + h.blocks + 1 + i);
    }
    HalfColumns sums;
    if (sums_out) sums = HalfColumns{c.at(sums_at), sums_out, accumulate ? 1 : 0};
    return launch_split_half(h.view, h.count, h.planes, h.status, h.blocks, sums, c.stream);
}

// One or two products, p[i] of operands x[i] and y[i], in one launch.
int run_halves(Call &c, GemmProblem *p, int count, const Halves &h, const HalfOperand *x, const HalfOperand *y, const char *const *labels) {
    for (int i = 0; i < count; ++i) {
        p[i].ha = &x[i];
        p[i].hb = &y[i];
        p[i].half_status = h.status + h.blocks;
        p[i].fast_tf32 = (c.flags & MNI_B200_PRECISION_TF32) != 0;
    }
    size_t bytes[2] = {0, 0};
    float *partial[2] = {nullptr, nullptr};
    gemm_halves_partial_bytes(p, count, c.gemm_sms(), bytes);
    for (int i = 0; i < count; ++i) {
        const size_t at = bytes[i] ? c.arena.reserve(bytes[i]) : 0;
        if (bytes[i] && !c.dry()) partial[i] = c.at(at);
    }
    if (c.plan_log) {
        std::string lines[2];
        gemm_halves_describe(p, count, c.gemm_sms(), lines);
        for (int i = 0; i < count; ++i) {
            if (labels) c.label = labels[i];
            c.note(lines[i]);
        }
    }
    if (c.dry()) return MNI_B200_OK;
    return launch_gemm_halves(p, count, partial, c.st->err_word, c.gemm_sms(), c.stream);
}

int zero_or_bias_fill(Call &c, float *out, int64_t rows, int64_t n, const float *bias, bool accumulate) {
    if (c.dry() || rows * n == 0) return MNI_B200_OK;
    if (!accumulate) MNI_CUDA(cudaMemsetAsync(out, 0, static_cast<size_t>(rows * n) * sizeof(float), c.stream));
    if (bias) return launch_add_bias(out, bias, out, rows, n, c.stream);
    return MNI_B200_OK;
}

struct Shapes {
    int64_t M, K, N;
    int64_t out_batch[MNI_B200_MAX_DIMS];
    int out_nb;
    int64_t batch, a_batch, b_batch;
};

int analyse(const mni_b200_view *a, const mni_b200_view *b, Shapes &s) {
    int rc = check_view(a, "a", 2);
    if (rc) return rc;
    rc = check_view(b, "b", 2);
    if (rc) return rc;
    s.M = a->shape[a->ndim - 2];
    s.K = a->shape[a->ndim - 1];
    s.N = b->shape[b->ndim - 1];
    if (b->shape[b->ndim - 2] != s.K)
        return fail(MNI_B200_ERR_INNER_DIM, "matmul inner dimensions must match: %lld vs %lld", (long long)s.K,
                    (long long)b->shape[b->ndim - 2]);
    s.out_nb = broadcast_shape(a->shape, a->ndim - 2, b->shape, b->ndim - 2, s.out_batch);
    if (s.out_nb < 0) return fail(MNI_B200_ERR_BROADCAST, "batch shapes are not broadcastable");
    s.batch = prod(s.out_batch, s.out_nb);
    s.a_batch = prod(a->shape, a->ndim - 2);
    s.b_batch = prod(b->shape, b->ndim - 2);
    return MNI_B200_OK;
}

bool aligned_weight(const Shapes &s, const mni_b200_view &w) {
    const int64_t s0 = w.stride[w.ndim - 2], s1 = w.stride[w.ndim - 1];
    return (reinterpret_cast<uintptr_t>(w.ptr) & 15) == 0 && (s1 == 1 ? s0 : s1) % 4 == 0 && (s1 == 1 ? s.N : s.K) % 4 == 0;
}
// Few rows against one weight, not forced onto another path.
bool rows_wanted(uint32_t flags, const Shapes &s, const mni_b200_view &w) {
    return (flags & (MNI_B200_FORCE_TENSOR_PATH | MNI_B200_FORCE_SKINNY_PATH | MNI_B200_FORCE_PACK)) == 0 &&
           ((flags >> 16) & 0xffu) == 0 && s.batch == 1 && s.a_batch == 1 && s.b_batch == 1 &&
           s.M <= (aligned_weight(s, w) ? kRowsAligned : kRowsUnaligned);
}
// Whether the product of `outs` outputs a row and a contraction of `total` is one the warp-level kernels take.
bool rows_take(const Shapes &s, const mni_b200_view &w, int64_t outs, int64_t total, int sm_count) {
    return rows_supported(s.M, outs, total, sm_count) &&
           (!aligned_weight(s, w) || total <= kRowsShort || (outs >= total && outs * total <= kRowsElements));
}

// What the one-launch f32 kernel would compute for a call.
enum TinyCall { kTinyForward, kTinyForwardGelu, kTinyGradA, kTinyGradB, kTinyGradBoth };

// Small enough for the one-launch f32 kernel: a single matrix product whose contraction (forward K, backward M and N), work and
// tiles are all small, operands readable along one of their dims.  MNI_B200_TINY overrides the limit on M * N * K (0: never).
bool tiny_wanted(const Call &c, TinyCall call, const Shapes &s, const mni_b200_view &a, const mni_b200_view &b, const mni_b200_view *dc) {
    auto readable = [](const mni_b200_view &v) { return v.stride[v.ndim - 1] == 1 || v.stride[v.ndim - 2] == 1; };
    const uint32_t forced = MNI_B200_FORCE_TENSOR_PATH | MNI_B200_FORCE_SKINNY_PATH | MNI_B200_FORCE_PACK | MNI_B200_PRECISION_TF32;
    if ((c.flags & forced) != 0 || ((c.flags >> 16) & 0xffu) != 0 || s.batch != 1 || s.a_batch != 1 || s.b_batch != 1 ||
        (dc ? std::max(s.M, s.N) : s.K) > (s.M <= 8 ? kTinyContractionFewRows : kTinyContraction) ||
        std::max({s.M, s.N, s.K}) > kTinyWork || s.M * s.N * s.K > env_int("MNI_B200_TINY", kTinyWork) || !readable(a) ||
        !readable(b) || (dc && !readable(*dc)))
        return false;
    const int64_t m = (s.M + 31) / 32, n = (s.N + 31) / 32, k = (s.K + 31) / 32;
    const bool da = call == kTinyGradA || call == kTinyGradBoth, db = call == kTinyGradB || call == kTinyGradBoth;
    const int64_t tiles = dc ? (da ? m * k : 0) + (db ? k * n : 0) : m * n;
    if (s.M > 8) {
        if (call == kTinyGradBoth) return tiles <= kTinyTilesBoth;
        const bool aligned_rows = (call == kTinyGradA ? s.K : s.N) % 4 == 0, exchanged = (call == kTinyGradB ? s.K : s.M) <= 64;
        return tiles <= (c.capturing && aligned_rows && !exchanged ? kTinyTilesCaptured : kTinyTiles);
    }
    if (tiles <= kTinyTilesFewest && (dc ? std::max(s.M, s.N) : s.K) <= 32) return true;
    const bool rows_unit = dc ? dc->stride[dc->ndim - 1] == 1 || s.N == 1 : a.stride[a.ndim - 1] == 1 || s.K == 1;
    const bool weight_aligned = (reinterpret_cast<uintptr_t>(b.ptr) & 15) == 0 && b.stride[b.ndim - 1] == 1 &&
                                b.stride[b.ndim - 2] % 4 == 0 && s.N % 4 == 0;
    switch (call) {
        case kTinyForward:
            return tiles <= (s.K > 64 ? kTinyTilesFewRows / 2 : kTinyTilesFewRows) &&
                   (!rows_unit || (weight_aligned && (s.M > 4 || s.K <= 64)));
        case kTinyForwardGelu: return tiles <= kTinyTilesFewRows;
        case kTinyGradA: return tiles <= kTinyTilesFewRows && !rows_unit;
        case kTinyGradB: return tiles <= kTinyTilesFewRows && (!c.capturing || s.M > 2);
        default:
            if (!c.capturing) return tiles <= kTinyTiles;
            return tiles <= (s.M > 4 ? kTinyTilesCaptured : s.M > 2 ? kTinyTilesFewRows / 2 : kTinyTilesFewest);
    }
}

// ------------------------------------------------------------------ forward
// a . b on the tensor path; `p` without its operands.
int forward_product(Call &c, const Shapes &s, const mni_b200_view *a, const mni_b200_view *b, GemmProblem &p) {
    HalfView probe;
    bool swapped;
    bool half = s.M > 128 && s.N > 128 && s.K >= 64 && half_possible(c, static_cast<double>(s.batch) * s.M * s.N * s.K) &&
                view_to_half(*a, probe, &swapped) && view_to_half(*b, probe, &swapped);
    if (half) {
        p.fast_tf32 = (c.flags & MNI_B200_PRECISION_TF32) != 0;
        half = half_pays(c, gemm_estimate_us(p, c.gemm_sms()) + gather_us(*a) + gather_us(*b), gemm_halves_estimate_us(&p, 1, c.gemm_sms()),
                         static_cast<double>(s.a_batch) * s.M * s.K + static_cast<double>(s.b_batch) * s.K * s.N);
    }
    const mni_b200_view *const a_given = a, *const b_given = b;
    int rc = MNI_B200_OK;
    if (!half || c.plan_log) {
        mni_b200_view packed[kMaxGathers];
        rc = pack_undescribable(c, {&a, &b}, packed);
        if (rc) return rc;
        rc = make_operand(*a, false, p.A);
        if (rc) return rc;
        rc = make_operand(*b, true, p.B);
        if (rc) return rc;
        p.A.batch = s.a_batch;
        p.B.batch = s.b_batch;
        rc = run_gemm(c, p);
        if (!half || rc) return rc;
        c.note("with scratch for 16-bit operands, instead of these:");
    }
    Halves h;
    rc = make_halves(c, {a_given, b_given}, h);
    if (rc) return rc;
    const HalfOperand x = h.operand(0, false), y = h.operand(1, true);
    return run_halves(c, &p, 1, h, &x, &y, nullptr);
}

int fwd_body(Call &c, const mni_b200_view *a, const mni_b200_view *b, float *out, const float *bias) {
    Shapes s;
    int rc = analyse(a, b, s);
    if (rc) return rc;
    if (!out && s.batch * s.M * s.N > 0) return fail(MNI_B200_ERR_ARG, "c is null");
    const bool accumulate = (c.flags & MNI_B200_ACCUMULATE_C) != 0;
    if (s.batch * s.M * s.N == 0) return MNI_B200_OK;
    if (s.K == 0) return zero_or_bias_fill(c, out, s.batch * s.M, s.N, bias, accumulate);

    if (!*c.label) c.label = "forward: ";
    if (tiny_wanted(c, kTinyForward, s, *a, *b, nullptr)) {
        c.note("small f32 kernel");
        if (c.dry()) return MNI_B200_OK;
        const TinyProduct p{a->ptr, b->ptr, out, bias, static_cast<int>(s.M), static_cast<int>(s.N), static_cast<int>(s.K),
                            accumulate ? 1 : 0, a->stride[a->ndim - 2], a->stride[a->ndim - 1], b->stride[b->ndim - 2],
                            b->stride[b->ndim - 1], s.N};
        return launch_tiny(&p, 1, nullptr, c.stream);
    }
    const bool want_skinny = (c.flags & MNI_B200_FORCE_SKINNY_PATH) != 0 ||
                             ((c.flags & MNI_B200_FORCE_TENSOR_PATH) == 0 && s.M <= skinny_fwd_row_limit(s.N));
    if (want_skinny && s.batch == 1 && skinny_fwd_supported(s.M, s.N, s.K)) {
        const int an = a->ndim, bn = b->ndim;
        const bool a_ok = a->stride[an - 1] == 1 || s.K == 1;
        const bool b_ok = (b->stride[bn - 1] == 1 || s.N == 1) && (b->stride[bn - 2] % 4 == 0 || s.K == 1) &&
                          (reinterpret_cast<uintptr_t>(b->ptr) & 15) == 0;
        if (a_ok && b_ok) {
            const size_t pbytes = skinny_fwd_partial_bytes(s.M, s.N, s.K, c.st->sm_count);
            const size_t poff = c.arena.reserve(pbytes);
            c.note("streaming (skinny) forward kernel");
            if (c.dry()) return MNI_B200_OK;
            const int64_t ldw = s.K == 1 ? round_up(s.N, 4) : b->stride[bn - 2];
            return launch_skinny_fwd(a->ptr, a->stride[an - 2], b->ptr, ldw, out, s.N, bias, accumulate, s.M, s.N,
                                     s.K, c.at(poff), c.st->sm_count, c.stream);
        }
    }

    if (rows_wanted(c.flags, s, *b) && rows_take(s, *b, s.N, s.K, c.st->sm_count) && (a->stride[a->ndim - 1] == 1 || s.K == 1)) {
        const int64_t ldx = a->stride[a->ndim - 2], sk = b->stride[b->ndim - 2], sn = b->stride[b->ndim - 1];
        if (sn == 1 || sk == 1) {                      // W as stored [K, N], or [N, K] seen through a transposing view
            c.note("streaming (few rows) forward kernel");
            if (c.dry()) return MNI_B200_OK;
            auto launch = sn == 1 ? launch_rows_fwd : launch_rows_bt_fwd;
            return launch(a->ptr, ldx, b->ptr, sn == 1 ? sk : sn, out, s.N, bias, accumulate, s.M, s.N, s.K,
                          c.st->sm_count, c.stream);
        }
    }

    GemmProblem p;
    p.M = s.M; p.N = s.N; p.K = s.K;
    p.batch = s.batch;
    p.fold = 1;
    p.C = out;
    p.ldc = s.N;
    p.c_bstride = s.M * s.N;
    p.bias = bias;
    p.accumulate = accumulate;
    return forward_product(c, s, a, b, p);
}

// Forward with the bias + GELU epilogue: pre = a . b (optional output), out = gelu(pre + bias).
int fwd_gelu_body(Call &c, const mni_b200_view *a, const mni_b200_view *b, const float *bias, float *pre,
                  float *out) {
    Shapes s;
    int rc = analyse(a, b, s);
    if (rc) return rc;
    const int64_t rows = s.batch * s.M;
    if (rows * s.N == 0) return MNI_B200_OK;
    if (!bias || !out) return fail(MNI_B200_ERR_ARG, "bias and out must not be null");
    const uint32_t saved_flags = c.flags;
    c.flags &= ~static_cast<uint32_t>(MNI_B200_ACCUMULATE_C);
    if (s.K > 0 && tiny_wanted(c, kTinyForwardGelu, s, *a, *b, nullptr)) {
        c.flags = saved_flags;
        if (c.dry()) return MNI_B200_OK;
        const TinyProduct p{a->ptr, b->ptr, pre, bias, static_cast<int>(s.M), static_cast<int>(s.N), static_cast<int>(s.K), 0,
                            a->stride[a->ndim - 2], a->stride[a->ndim - 1], b->stride[b->ndim - 2], b->stride[b->ndim - 1], s.N, out};
        return launch_tiny(&p, 1, nullptr, c.stream);
    }
    const bool skinny = (c.flags & MNI_B200_FORCE_SKINNY_PATH) != 0 ||
                        ((c.flags & MNI_B200_FORCE_TENSOR_PATH) == 0 && s.M <= skinny_fwd_row_limit(s.N));
    if (s.K > 0 && !skinny) {
        GemmProblem p;
        p.M = s.M; p.N = s.N; p.K = s.K;
        p.batch = s.batch;
        p.C = pre; p.D = out;
        p.ldc = s.N; p.c_bstride = s.M * s.N;
        p.bias = bias;
        p.fast_tf32 = (c.flags & MNI_B200_PRECISION_TF32) != 0;
        p.force_splits = static_cast<int>((c.flags >> 16) & 0xffu);
        if (gemm_tc_can_fuse_activation(p, c.gemm_sms())) {
            rc = forward_product(c, s, a, b, p);
            c.flags = saved_flags;
            return rc;
        }
    }
    // Not fusable (split-K, skinny rows, unaligned rows): the product first, then the pointwise kernel.
    float *tmp = pre;
    size_t off = 0;
    if (!tmp) off = c.arena.reserve(static_cast<size_t>(rows * s.N) * sizeof(float));
    if (!tmp && !c.dry()) tmp = c.at(off);
    rc = fwd_body(c, a, b, c.dry() && !tmp ? reinterpret_cast<float *>(static_cast<uintptr_t>(256)) : tmp, nullptr);
    c.flags = saved_flags;
    if (rc || c.dry()) return rc;
    return launch_bias_gelu(tmp, bias, out, rows, s.N, c.stream);
}

// ------------------------------------------------------------------ backward
// Whether the target's batch dims, right-aligned against ob, are all equal to it (`same`), or hold a single matrix: then
// one product writes the gradient, with no unbroadcast after it.
bool single_product(const int64_t *ob, int onb, const mni_b200_view &target, bool *same) {
    const int tnb = target.ndim - 2;
    *same = tnb <= onb;
    for (int i = 0; *same && i < onb; ++i) {
        const int64_t td = i < onb - tnb ? 1 : target.shape[i - (onb - tnb)];
        if (td != ob[i]) *same = false;
    }
    return *same || prod(ob, onb) == 1 || prod(target.shape, tnb) == 1;
}

// One gradient: G[ob.., R, Cn] = X . Y (a GEMM over `kdim`) reduced to `target`'s shape.
//   X supplies the rows, Y the columns; both already as Operands with flat batch counts.
int grad_gemm(Call &c, Operand X, Operand Y, int64_t R, int64_t Cn, int64_t kdim, const int64_t *ob, int onb,
              const mni_b200_view &target, float *out, bool accumulate) {
    const int64_t obatch = prod(ob, onb);
    const int64_t tbatch = prod(target.shape, target.ndim - 2);
    bool same = false;
    single_product(ob, onb, target, &same);
    GemmProblem p;
    p.A = X; p.B = Y;
    p.M = R; p.N = Cn; p.K = kdim;
    p.bias = nullptr;
    if (same || obatch == 1) {
        p.batch = obatch; p.fold = 1;
        p.C = out; p.ldc = Cn; p.c_bstride = R * Cn; p.accumulate = accumulate;
        return run_gemm(c, p);
    }
    if (tbatch == 1) {
        // The operand was broadcast over every batch: sum the batches inside the contraction.
        p.batch = 1; p.fold = obatch;
        p.C = out; p.ldc = Cn; p.c_bstride = R * Cn; p.accumulate = accumulate;
        return run_gemm(c, p);
    }
    // Partial broadcast: full batched product into scratch, then the device-side unbroadcast.
    const size_t bytes = static_cast<size_t>(obatch * R * Cn) * sizeof(float);
    const size_t off = c.arena.reserve(bytes);
    p.batch = obatch; p.fold = 1;
    p.C = c.dry() ? nullptr : c.at(off);
    p.ldc = Cn; p.c_bstride = R * Cn; p.accumulate = false;
    int rc = run_gemm(c, p);
    c.note("sum over the broadcast batch dims (unbroadcast kernel)");
    if (rc || c.dry()) return rc;
    int64_t gshape[MNI_B200_MAX_DIMS + 2];
    for (int i = 0; i < onb; ++i) gshape[i] = ob[i];
    gshape[onb] = R; gshape[onb + 1] = Cn;
    return launch_unbroadcast(c.at(off), gshape, onb + 2, target.shape, target.ndim, out, accumulate, c.stream);
}

// The gradients on the tensor path as products of 16-bit planes, the one of the longer contraction first: units that take
// longer are better dealt out early.
struct HalfGrads {
    GemmProblem p[2];
    bool is_a[2];                      // grad_a = dc . b^T, or grad_b = a^T . dc
    int count = 0;
};
// Whether they are computed so: one product each, of operands that have planes, and worth it.
bool bwd_half_wanted(const Call &c, const Shapes &s, const mni_b200_view &a, const mni_b200_view &b, const mni_b200_view &dc, bool da,
                     bool db, int64_t g_batch, double work, HalfGrads &g) {
    if ((!da && !db) || s.M < 64 || s.N < 64 || s.K <= 128 || (da && s.M <= 128) || (db && s.N <= 128) || !half_possible(c, work)) return false;
    HalfView probe;
    bool swapped;
    if (!view_to_half(dc, probe, &swapped)) return false;
    double elements = static_cast<double>(g_batch) * s.M * s.N, f32_us = 0, beside_us = 0, gathers_us = gather_us(dc);
    const int all = c.gemm_sms(1), halved = c.gemm_sms(2);
    auto product = [&](const mni_b200_view &other, const mni_b200_view &target, int64_t rows, int64_t cols, int64_t k, bool is_a) {
        int64_t ob[MNI_B200_MAX_DIMS];
        bool same;
        const int nb = broadcast_shape(other.shape, other.ndim - 2, dc.shape, dc.ndim - 2, ob);
        if (nb < 0 || !single_product(ob, nb, target, &same) || !view_to_half(other, probe, &swapped)) return false;
        const int64_t count = prod(ob, nb);
        g.is_a[g.count] = is_a;
        GemmProblem &p = g.p[g.count++];
        p.M = rows; p.N = cols; p.K = k;
        p.batch = same ? count : 1;
        p.fold = same ? 1 : count;
        p.ldc = cols; p.c_bstride = rows * cols;
        p.fast_tf32 = (c.flags & MNI_B200_PRECISION_TF32) != 0;
        f32_us += gemm_estimate_us(p, all);
        gathers_us += gather_us(other);
        beside_us = std::max(beside_us, 1.25 * gemm_estimate_us(p, halved));   // beside one another they are that much slower (half_pays)
        elements += static_cast<double>(prod(other.shape, other.ndim));
        return true;
    };
    if (da && !product(b, a, s.M, s.K, s.N, true)) return false;
    if (db && !product(a, b, s.K, s.N, s.M, false)) return false;
    if (g.count == 2 && g.p[1].K * g.p[1].fold > g.p[0].K * g.p[0].fold) {
        std::swap(g.p[0], g.p[1]);
        std::swap(g.is_a[0], g.is_a[1]);
    }
    return half_pays(c, gathers_us + (da && db ? std::min(f32_us, beside_us) : f32_us), gemm_halves_estimate_us(g.p, g.count, all), elements);
}

int bwd_body(Call &c, const mni_b200_view *a, const mni_b200_view *b, const mni_b200_view *dc, float *da,
             float *db, float *dbias) {
    Shapes s;
    int rc = analyse(a, b, s);
    if (rc) return rc;
    rc = check_view(dc, "dc", 2);
    if (rc) return rc;
    const int gn = dc->ndim;
    if (dc->shape[gn - 2] != s.M || dc->shape[gn - 1] != s.N)
        return fail(MNI_B200_ERR_ARG, "dc is [.., %lld, %lld] but the forward output is [.., %lld, %lld]",
                    (long long)dc->shape[gn - 2], (long long)dc->shape[gn - 1], (long long)s.M, (long long)s.N);
    const int64_t g_batch = prod(dc->shape, gn - 2);
    const bool acc_da = (c.flags & MNI_B200_ACCUMULATE_DA) != 0;
    const bool acc_db = (c.flags & MNI_B200_ACCUMULATE_DB) != 0;
    const bool acc_dbias = (c.flags & MNI_B200_ACCUMULATE_DBIAS) != 0;
    const int64_t a_elems = s.a_batch * s.M * s.K, b_elems = s.b_batch * s.K * s.N;

    // Which kernel each gradient takes.
    const bool da_wanted = da && a_elems > 0 && s.N > 0 && g_batch > 0;
    const bool db_wanted = db && b_elems > 0 && s.M > 0 && g_batch > 0;
    if (g_batch == 1 && s.M > 0 && s.N > 0 && s.K > 0 && (da || db) && (!dbias || dc->stride[gn - 1] == 1) &&
        tiny_wanted(c, da && db ? kTinyGradBoth : da ? kTinyGradA : kTinyGradB, s, *a, *b, dc)) {
        c.label = "grad_a, grad_b, grad_bias: ";
        c.note("small f32 kernel");
        c.label = "";
        if (c.dry()) return MNI_B200_OK;
        const int M = static_cast<int>(s.M), N = static_cast<int>(s.N), K = static_cast<int>(s.K);
        const long long a_m = a->stride[a->ndim - 2], a_k = a->stride[a->ndim - 1], b_k = b->stride[b->ndim - 2],
                        b_n = b->stride[b->ndim - 1], g_m = dc->stride[gn - 2], g_n = dc->stride[gn - 1];
        TinyProduct p[kMaxTiny];
        int count = 0;
        if (da) p[count++] = TinyProduct{dc->ptr, b->ptr, da, nullptr, M, K, N, acc_da ? 1 : 0, g_m, g_n, b_n, b_k, s.K};
        if (db) p[count++] = TinyProduct{a->ptr, dc->ptr, db, nullptr, K, N, M, acc_db ? 1 : 0, a_k, a_m, g_m, g_n, s.N};
        const TinyColumns columns{dc->ptr, dbias, g_m, M, N, acc_dbias ? 1 : 0};
        return launch_tiny(p, count, dbias ? &columns : nullptr, c.stream);
    }
    const bool skinny_dx = da_wanted &&
                           ((c.flags & MNI_B200_FORCE_SKINNY_PATH) != 0 ||
                            ((c.flags & MNI_B200_FORCE_TENSOR_PATH) == 0 && s.M <= kSkinnyDxRows)) &&
                           s.batch == 1 && g_batch == 1 && s.a_batch == 1 && s.b_batch == 1 &&
                           dc->stride[gn - 1] == 1 && b->stride[b->ndim - 1] == 1 && s.K > 1 &&
                           skinny_dx_supported(dc->ptr, dc->stride[gn - 2], b->ptr, b->stride[b->ndim - 2], s.M, s.N);
    const bool rows_ok = rows_wanted(c.flags, s, *b) && g_batch == 1 && (dc->stride[gn - 1] == 1 || s.N == 1);
    // ... and those of the remaining few-row products that stream the weight through the warp-level kernels
    const int64_t b_sk = b->stride[b->ndim - 2], b_sn = b->stride[b->ndim - 1];
    const bool rows_dx = da_wanted && !skinny_dx && rows_ok && rows_take(s, *b, s.K, s.N, c.st->sm_count) && (b_sn == 1 || b_sk == 1);
    const bool skinny_dw = db_wanted &&
                           ((c.flags & MNI_B200_FORCE_SKINNY_PATH) != 0 || rows_ok ||
                            ((c.flags & MNI_B200_FORCE_TENSOR_PATH) == 0 && s.M <= kSkinnyDwRows)) &&
                           s.batch == 1 && g_batch == 1 && s.M <= 16 && (a->stride[a->ndim - 1] == 1 || s.K == 1) &&
                           (dc->stride[gn - 1] == 1 || s.N == 1);
    const bool streamed_dx = skinny_dx || rows_dx, streamed_dw = skinny_dw;

    // grad_a and grad_b do not depend on each other.  grad_b of a small problem goes to the library's side stream
    // next to grad_a and is joined before returning (event fork / join, also valid under stream capture).  The
    // column sums of the bias gradient are HBM-bound and always go to the side stream, where they run beside the
    // tensor-bound products instead of in front of them.
    // Two tensor-core products of a small problem are launched back to back on ONE stream as an independent pair
    // (GemmProblem::dep_mode: the second starts as soon as every CTA of the first has passed its own dependency wait), then
    // their finishes.  Under stream capture they go to two branches of the graph instead.  Measured: events between
    // streams cost an eager call 4-20 us (16 rows x 4096^2: 87 -> 66 us a step; 512^3: 35.0 -> 31.6) but a graph nothing
    // (512^3: pair 32.1, branches 26.7).  MNI_B200_BWD_PAIR=0 / 1 never / always pairs.
    const double work = static_cast<double>(s.M) * static_cast<double>(s.N) * static_cast<double>(s.K) *
                        static_cast<double>(std::max<int64_t>(g_batch, 1));
    // The decisions are the same in the sizing pass and in the real pass (they change the plans, hence the scratch);
    // only the stream operations are skipped while sizing.
    const bool side_on = env_flag("MNI_B200_BWD_OVERLAP", 1);
    const bool two_tensor = da_wanted && db_wanted && !streamed_dx && !streamed_dw;
    const bool small = work > 0 && work <= overlap_work_limit();
    bool pairable = false, beside = small, b_first = false;
    if (side_on && two_tensor) {
        int64_t oa[MNI_B200_MAX_DIMS], ob[MNI_B200_MAX_DIMS];
        bool same;
        const int na = broadcast_shape(dc->shape, gn - 2, b->shape, b->ndim - 2, oa);
        const int nb = broadcast_shape(a->shape, a->ndim - 2, dc->shape, gn - 2, ob);
        pairable = na >= 0 && nb >= 0 && single_product(oa, na, *a, &same) && single_product(ob, nb, *b, &same);
        if (pairable) {
            auto problem = [&](int64_t rows, int64_t cols, int64_t k, const int64_t *batch_dims, int nd, const mni_b200_view &target,
                               float *out) {
                bool is_same;
                single_product(batch_dims, nd, target, &is_same);
                const int64_t count = prod(batch_dims, nd);
                GemmProblem p;
                p.M = rows; p.N = cols; p.K = k;
                p.batch = is_same ? count : 1;
                p.fold = is_same ? 1 : count;
                p.C = out; p.ldc = cols; p.c_bstride = rows * cols;
                p.fast_tf32 = (c.flags & MNI_B200_PRECISION_TF32) != 0;
                p.force_splits = static_cast<int>((c.flags >> 16) & 0xffu);
                return p;
            };
            const GemmProblem pa = problem(s.M, s.K, s.N, oa, na, *a, da), pb = problem(s.K, s.N, s.M, ob, nb, *b, db);
            GemmProblem pa_half = pa, pb_half = pb;
            pa_half.beside = pb_half.beside = true;
            const int all = c.gemm_sms();
            c.sm_share = 2;
            const int half = c.gemm_sms();
            c.sm_share = 1;
            if (!small) {
                // Larger products go side by side where the cost model says so by a margin: where one of them, or both, would
                // leave SMs idle on its own or need a split of the contraction to fill them (2048 x 3072 x 768: 97.6 -> 81.4 us).
                const double whole_a = gemm_tc_estimate_us(pa, all), whole_b = gemm_tc_estimate_us(pb, all);
                const double half_a = gemm_tc_estimate_us(pa_half, half), half_b = gemm_tc_estimate_us(pb_half, half);
                beside = whole_a > 0 && whole_b > 0 && half_a > 0 && half_b > 0 && std::max(half_a, half_b) < 0.9 * (whole_a + whole_b);
            }
            // CTA pairs take both SMs of a unit, lone CTAs are dealt out one to a unit: launched first, these would leave
            // the pairs hardly a whole unit until they end (16 rows x 4096^2, grad_b in pairs after grad_a: 47 us against 37).
            b_first = beside && !gemm_tc_uses_pairs(pa_half, half) && gemm_tc_uses_pairs(pb_half, half);
        }
    }
    const int pair_env = env_int("MNI_B200_BWD_PAIR", -1);
    const bool pair = pairable && (pair_env > 0 || (pair_env < 0 && beside && !c.capturing));
    // Streamed gradients that each keep HBM busy on their own run one after the other: of one row against a very large weight
    // (8192 x 8192 97 us against 111 side by side, 4096 x 20000 120 / 137; four rows 120 / 111), and the streaming dW of 9 to 12
    // rows with whichever kernel computes dx (4096 x 4096 40 / 44, 5504 x 7680 87 / 92, 4096 x 20000 148 / 164; 15 rows 49 / 50).
    const bool in_turn = skinny_dw && da_wanted && ((s.M == 1 && s.K * s.N >= (int64_t{1} << 26)) ||
                                                    (s.M > 8 && s.M <= 12 && s.K * s.N >= (int64_t{1} << 24)));
    const bool overlap = side_on && !pair && da && db && a_elems > 0 && b_elems > 0 && beside && !in_turn;
    const bool side_dbias = side_on && dbias && (da || db) && work > 0;
    // Two tensor-core products side by side: each persistent grid is planned for half of the SMs, so that both are
    // resident at once instead of the second queueing behind the first's CTAs (measured under graph replay: 512^3
    // 29.2 -> 24.6 us per step, 1024^3 55.3 -> 45.3 us).
    const bool share_sms = (overlap || pair) && beside && two_tensor && env_flag("MNI_B200_BWD_SHARE_SMS", 1);
    if (share_sms) c.sm_share = 2;
    cudaStream_t const main_stream = c.stream;
    // Operands of the tensor path that have to be gathered: once each, before the streams part.
    mni_b200_view packed[kMaxGathers];
    const bool da_tensor = da_wanted && !streamed_dx, db_tensor = db_wanted && !streamed_dw;
    const mni_b200_view *const dc_given = dc, *const a_given = a, *const b_given = b;
    auto pack = [&]() -> int {
        c.label = "operands: ";
        int r = MNI_B200_OK;
        if (da_tensor && db_tensor) r = pack_undescribable(c, {&dc, &b, &a}, packed);
        else if (da_tensor) r = pack_undescribable(c, {&dc, &b}, packed);
        else if (db_tensor) r = pack_undescribable(c, {&dc, &a}, packed);
        c.label = "";
        return r;
    };
    // From 16-bit planes, in one launch on all SMs, instead of everything above and below but the column sums.
    HalfGrads half_grads;
    const bool half = bwd_half_wanted(c, s, *a, *b, *dc, da_tensor, db_tensor, g_batch, work, half_grads), halves_now = half && !c.plan_log;
    if (halves_now) c.sm_share = 1;
    else rc = pack();
    if (rc) return rc;
    // ... whose pass over dc can make them too
    const bool halves_dbias = halves_now && dbias && dc->stride[gn - 1] == 1;
    const bool fork = !c.dry() && ((overlap && !halves_now) || (side_dbias && !halves_dbias));
    if (fork) {
        MNI_CUDA(cudaEventRecord(c.st->ev_fork, main_stream));
        MNI_CUDA(cudaStreamWaitEvent(c.st->side, c.st->ev_fork, 0));
    }
    struct Join {      // joins the side stream on every exit path once it has been forked
        Call &c; cudaStream_t main; bool on;
        ~Join() {
            c.flag_bank = 0;
            c.dep_mode = 0;
            c.defer = nullptr;
            c.sm_share = 1;
            c.label = "";
            if (!on) return;
            c.stream = main;
            if (cudaEventRecord(c.st->ev_join, c.st->side) == cudaSuccess) cudaStreamWaitEvent(main, c.st->ev_join, 0);
        }
    } join{c, main_stream, fork};

    if (share_sms) c.note("grad_a and grad_b side by side, each planned for half of the SMs");
    else if (overlap) c.note("grad_b on the side stream beside grad_a");
    if (dbias && !halves_dbias) {
        // Column sums over every row of dc (ops/elementwise.rs:224-229 via utils::unbroadcast).
        c.label = "grad_bias: ";
        if (side_dbias && !c.dry()) c.stream = c.st->side;
        const int64_t rows = g_batch * s.M;
        if (rows == 0 || s.N == 0) {
            rc = zero_or_bias_fill(c, dbias, 1, s.N, nullptr, acc_dbias);
            if (rc) return rc;
        } else {
            // a gathered dc serves here too: its rows follow one another at the padded pitch
            mni_b200_view flat;
            const mni_b200_view *rows_of = dc;
            if (dc == dc_given) {
                bool contiguous = true;
                int64_t expect = 1;
                for (int d = gn - 1; d >= 0; --d) {
                    if (dc->shape[d] != 1 && dc->stride[d] != expect) contiguous = false;
                    expect *= dc->shape[d];
                }
                const mni_b200_view **use = &rows_of;
                if (!contiguous) rc = pack_views(c, &use, &flat, 1);
                if (rc) return rc;
            }
            const float *src = rows_of->ptr;
            const int64_t ld = rows_of == dc_given ? s.N : rows_of->stride[1];
            const size_t pbytes = colsum_partial_bytes(rows, s.N, c.st->sm_count);
            const size_t poff = c.arena.reserve(pbytes);
            c.note(side_dbias ? "column sums, on the side stream" : "column sums");
            if (!c.dry()) {
                rc = launch_colsum(src, ld, nullptr, dbias, rows, s.N, acc_dbias, c.at(poff), c.st->sm_count, c.stream);
                if (rc) return rc;
            }
        }
    }

    c.stream = main_stream;

    auto halves = [&]() -> int {
        Halves h;
        c.label = "gradients: ";
        if (c.plan_log) c.note("with scratch for 16-bit operands, instead of these:");
        float *const sums = halves_dbias ? dbias : nullptr;
        int r = da_tensor && db_tensor ? make_halves(c, {dc_given, b_given, a_given}, h, sums, acc_dbias)
                : da_tensor            ? make_halves(c, {dc_given, b_given}, h, sums, acc_dbias)
                                       : make_halves(c, {dc_given, a_given}, h, sums, acc_dbias);
        if (r) return r;
        HalfOperand x[2], y[2];
        const char *labels[2];
        for (int i = 0; i < half_grads.count; ++i) {
            const bool is_a = half_grads.is_a[i];
            labels[i] = is_a ? "grad_a: " : "grad_b: ";
            x[i] = is_a ? h.operand(0, false) : h.operand(da_tensor ? 2 : 1, true);
            y[i] = is_a ? h.operand(1, false) : h.operand(0, true);
            half_grads.p[i].C = is_a ? da : db;
            half_grads.p[i].accumulate = is_a ? acc_da : acc_db;
        }
        r = run_halves(c, half_grads.p, half_grads.count, h, x, y, labels);
        return r;
    };
    if (halves_now) return halves();

    GemmFinish finish[2];              // of a pair: launched after both products
    // What the first (0) or second (1) product issued is launched with: an independent pair on one stream, or the second
    // on the side stream.
    auto place = [&](int at) {
        c.dep_mode = pair ? at + 1 : 0;
        c.defer = pair ? &finish[at] : nullptr;
        if (at == 1 && overlap && !c.dry()) c.stream = c.st->side;
        c.flag_bank = at == 1 && (overlap || pair) ? 1 : 0;
    };

    // grad_a = unbroadcast(dc . b^T, a.shape)   (ops/matmul.rs:231-240)
    auto grad_a = [&](int at) -> int {
        c.label = "grad_a: ";
        place(at);
        if (!da || a_elems == 0) return MNI_B200_OK;
        if (!da_wanted) {
            rc = zero_or_bias_fill(c, da, a_elems, 1, nullptr, acc_da);
            if (rc) return rc;
        } else if (skinny_dx) {
            c.note("streaming (skinny) input-gradient kernel");
            if (!c.dry()) {
                rc = launch_skinny_dx(dc_given->ptr, dc_given->stride[gn - 2], b_given->ptr, b_given->stride[b_given->ndim - 2], da, s.K, acc_da,
                                      s.M, s.N, s.K, !overlap, c.stream);
                if (rc) return rc;
            }
        } else if (rows_dx) {
            c.note("streaming (few rows) input-gradient kernel");
            if (!c.dry()) {
                auto launch = b_sn == 1 ? launch_rows_dx : launch_rows_bt_dx;
                rc = launch(dc_given->ptr, dc_given->stride[gn - 2], b_given->ptr, b_sn == 1 ? b_sk : b_sn, da, s.K, nullptr, acc_da,
                            s.M, s.N, s.K, c.st->sm_count, c.stream);
                if (rc) return rc;
            }
        } else {
            int64_t ob[MNI_B200_MAX_DIMS];
            const int onb = broadcast_shape(dc_given->shape, gn - 2, b_given->shape, b_given->ndim - 2, ob);
            if (onb < 0) return fail(MNI_B200_ERR_BROADCAST, "dc and b batch shapes are not broadcastable");
            Operand X, Y;
            rc = make_operand(*dc, false, X);   // rows M, contraction N
            if (rc) return rc;
            rc = make_operand(*b, false, Y);    // rows K, contraction N
            if (rc) return rc;
            X.batch = g_batch;
            Y.batch = s.b_batch;
            rc = grad_gemm(c, X, Y, s.M, s.K, s.N, ob, onb, *a_given, da, acc_da);
            if (rc) return rc;
        }
        return MNI_B200_OK;
    };

    // grad_b = unbroadcast(a^T . dc, b.shape)   (ops/matmul.rs:242-251)
    auto grad_b = [&](int at) -> int {
        c.label = "grad_b: ";
        place(at);
        if (!db || b_elems == 0) return MNI_B200_OK;
        if (!db_wanted) {
            rc = zero_or_bias_fill(c, db, b_elems, 1, nullptr, acc_db);
            if (rc) return rc;
        } else if (skinny_dw) {
            c.note("streaming (skinny) weight-gradient kernel");
            if (!c.dry()) {
                rc = launch_skinny_dw(a_given->ptr, a_given->stride[a_given->ndim - 2], dc_given->ptr, dc_given->stride[gn - 2], db, s.N, acc_db,
                                      s.M, s.N, s.K, c.stream);
                if (rc) return rc;
            }
        } else {
            int64_t ob[MNI_B200_MAX_DIMS];
            const int onb = broadcast_shape(a_given->shape, a_given->ndim - 2, dc_given->shape, gn - 2, ob);
            if (onb < 0) return fail(MNI_B200_ERR_BROADCAST, "a and dc batch shapes are not broadcastable");
            Operand X, Y;
            rc = make_operand(*a, true, X);     // rows K, contraction M
            if (rc) return rc;
            rc = make_operand(*dc, true, Y);    // rows N, contraction M
            if (rc) return rc;
            X.batch = s.a_batch;
            Y.batch = g_batch;
            rc = grad_gemm(c, X, Y, s.K, s.N, s.M, ob, onb, *b_given, db, acc_db);
            if (rc) return rc;
        }
        return MNI_B200_OK;
    };
    rc = b_first ? grad_b(0) : grad_a(0);
    if (rc == MNI_B200_OK) rc = b_first ? grad_a(1) : grad_b(1);
    c.dep_mode = 0;
    const bool both = finish[0] && finish[1];
    if (rc == MNI_B200_OK && finish[0]) rc = finish[0](both ? 1 : 0, c.stream);
    if (rc == MNI_B200_OK && finish[1]) rc = finish[1](both ? 2 : 0, c.stream);
    if (rc == MNI_B200_OK && half) {
        c.sm_share = 1;
        rc = halves();
    }
    return rc;
}

// Runs `body` twice: a dry pass that sizes the scratch, then the real pass.
template <class Body>
int with_scratch(uint32_t flags, void *stream, Body body) {
    EnvScope env;
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(st->mu);
    const bool capturing = stream_is_capturing(static_cast<cudaStream_t>(stream));
    Call real;
    real.capturing = capturing;
    real.st = st; real.arena.st = st; real.arena.dry = false; real.stream = static_cast<cudaStream_t>(stream); real.flags = flags;
    size_t sized = 0;
    while (true) {
        Call dry;
        dry.capturing = capturing;
        dry.no_half = real.no_half;
        dry.st = st; dry.arena.st = st; dry.arena.dry = true; dry.stream = static_cast<cudaStream_t>(stream); dry.flags = flags;
        rc = body(dry);
        if (rc) return rc;
        sized = dry.arena.used;
        if (sized == 0) break;
        // Not what would have to be allocated in a capture, which that would end, nor what could not be had before.
        if (dry.used_half && !st->user_ws && sized > st->ws_bytes && (capturing || scratch_refused(*st, sized))) {
            real.no_half = true;
            continue;
        }
        rc = scratch_base(*st, sized, real.stream, &real.base);
        if (rc == MNI_B200_OK) break;
        // Scratch for the operands' planes cannot be had: the call goes without them, as it needs little or none then.
        if (!dry.used_half || real.no_half) return rc;
        if (!st->user_ws) note_refused(*st, sized);
        real.no_half = true;
    }
    rc = body(real);
    // Both passes must have planned the same launches: a real pass that asked for more scratch than was sized
    // would have written past it.
    if (rc == MNI_B200_OK && real.arena.used > sized)
        return fail(MNI_B200_ERR_WORKSPACE, "internal: the call used %zu bytes of scratch, %zu were sized", real.arena.used, sized);
    return rc;
}

}  // namespace

int device_sm_count() {
    static std::atomic<int> cache[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

bool pdl_enabled() {
    static const bool on = env_flag("MNI_B200_PDL", 1);
    return on;
}

// The switches found by the innermost open EnvScope of this thread: pointers into the environment block, valid while
// the call runs under the same rule as getenv's results.
namespace {
constexpr int kMaxSwitches = 48;
struct EnvSnapshot {
    int depth = 0, count = 0;             // count > kMaxSwitches: more than fit, and the environment is asked as outside a scope
    const char *entry[kMaxSwitches];      // "NAME=value"
};
thread_local EnvSnapshot t_env;
}  // namespace

EnvScope::EnvScope() {
    if (t_env.depth++ != 0) return;
    t_env.count = 0;
    for (char **e = environ; e && *e; ++e)
        if ((*e)[0] == 'M' && strncmp(*e, "MNI_B200_", 9) == 0) {
            if (t_env.count == kMaxSwitches) { ++t_env.count; break; }
            t_env.entry[t_env.count++] = *e;
        }
}
EnvScope::~EnvScope() { --t_env.depth; }

const char *env_value(const char *name) {
    const char *v = nullptr;
    if (t_env.depth == 0 || t_env.count > kMaxSwitches) {
        v = getenv(name);
    } else {
        for (int i = 0; i < t_env.count; ++i) {
            const size_t n = strlen(name);
            if (strncmp(t_env.entry[i], name, n) == 0 && t_env.entry[i][n] == '=') { v = t_env.entry[i] + n + 1; break; }
        }
    }
    return v && *v ? v : nullptr;
}
int env_int(const char *name, int dflt) {
    const char *v = env_value(name);
    return v ? atoi(v) : dflt;
}

int fail(int status, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(t_error, sizeof(t_error), fmt, ap);
    va_end(ap);
    return status;
}

}  // namespace mni

using namespace mni;

extern "C" {

int mni_b200_version(void) { return 100; }

const char *mni_b200_last_error(void) { return t_error; }

uint64_t mni_b200_launch_count(void) { return g_launches.load(); }

int mni_b200_matmul_fwd(const mni_b200_view *a, const mni_b200_view *b, float *c, const float *bias,
                        uint32_t flags, void *stream) {
    Shapes s;   // argument errors are reported before any device is touched
    int rc = analyse(a, b, s);
    if (rc) return rc;
    return with_scratch(flags, stream, [&](Call &call) { return fwd_body(call, a, b, c, bias); });
}

int mni_b200_matmul_bias_gelu_fwd(const mni_b200_view *a, const mni_b200_view *b, const float *bias, float *pre,
                                  float *out, uint32_t flags, void *stream) {
    Shapes s;
    int rc = analyse(a, b, s);
    if (rc) return rc;
    return with_scratch(flags, stream, [&](Call &call) { return fwd_gelu_body(call, a, b, bias, pre, out); });
}

int mni_b200_matmul_bwd(const mni_b200_view *a, const mni_b200_view *b, const mni_b200_view *dc, float *da,
                        float *db, float *dbias, uint32_t flags, void *stream) {
    Shapes s;
    int rc = analyse(a, b, s);
    if (rc) return rc;
    rc = check_view(dc, "dc", 2);
    if (rc) return rc;
    if (dc->shape[dc->ndim - 2] != s.M || dc->shape[dc->ndim - 1] != s.N)
        return fail(MNI_B200_ERR_ARG, "dc is [.., %lld, %lld] but the forward output is [.., %lld, %lld]",
                    (long long)dc->shape[dc->ndim - 2], (long long)dc->shape[dc->ndim - 1], (long long)s.M,
                    (long long)s.N);
    return with_scratch(flags, stream, [&](Call &call) { return bwd_body(call, a, b, dc, da, db, dbias); });
}

int mni_b200_add_bias(const float *y, const float *bias, float *out, int64_t rows, int64_t n, void *stream) {
    if (rows < 0 || n < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (rows * n == 0) return MNI_B200_OK;
    if (!y || !bias || !out) return fail(MNI_B200_ERR_ARG, "null pointer");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    return launch_add_bias(y, bias, out, rows, n, static_cast<cudaStream_t>(stream));
}

int mni_b200_add_bias_bwd(const float *dy, float *d_y, float *dbias, int64_t rows, int64_t n, uint32_t flags,
                          void *stream) {
    if (rows < 0 || n < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (!dy && rows * n > 0) return fail(MNI_B200_ERR_ARG, "dy is null");
    return with_scratch(flags, stream, [&](Call &c) -> int {
        if (!dbias || n == 0) return c.dry() ? static_cast<int>(MNI_B200_OK) : launch_copy(dy, d_y, rows * n, c.stream);
        const bool acc = (flags & MNI_B200_ACCUMULATE_DBIAS) != 0;
        if (rows == 0) return zero_or_bias_fill(c, dbias, 1, n, nullptr, acc);
        const size_t poff = c.arena.reserve(colsum_partial_bytes(rows, n, c.st->sm_count));
        if (c.dry()) return MNI_B200_OK;
        return launch_colsum(dy, n, d_y != dy ? d_y : nullptr, dbias, rows, n, acc, c.at(poff), c.st->sm_count, c.stream);
    });
}

int mni_b200_bias_gelu(const float *x, const float *bias, float *out, int64_t rows, int64_t n, void *stream) {
    if (rows < 0 || n < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (rows * n == 0) return MNI_B200_OK;
    if (!x || !bias || !out) return fail(MNI_B200_ERR_ARG, "null pointer");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    return launch_bias_gelu(x, bias, out, rows, n, static_cast<cudaStream_t>(stream));
}

int mni_b200_bias_gelu_bwd(const float *grad, const float *x, const float *bias, float *dx, float *dbias,
                           int64_t rows, int64_t n, uint32_t flags, void *stream) {
    if (rows < 0 || n < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (rows * n > 0 && (!grad || !x || !bias || !dx)) return fail(MNI_B200_ERR_ARG, "null pointer");
    if (n > 0 && !dbias) return fail(MNI_B200_ERR_ARG, "dbias is null");
    return with_scratch(flags, stream, [&](Call &c) -> int {
        const bool acc = (flags & MNI_B200_ACCUMULATE_DBIAS) != 0;
        if (n == 0) return MNI_B200_OK;
        if (rows == 0) return zero_or_bias_fill(c, dbias, 1, n, nullptr, acc);
        const size_t poff = c.arena.reserve(colsum_partial_bytes(rows, n, c.st->sm_count));
        if (c.dry()) return MNI_B200_OK;
        return launch_bias_gelu_bwd(grad, x, bias, dx, dbias, rows, n, acc, c.at(poff), c.st->sm_count, c.stream);
    });
}

static int softmax_args(const void *p0, const void *p1, const void *p2, int64_t outer, int64_t dim, int64_t inner) {
    if (outer < 0 || dim < 0 || inner < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (outer == 0 || dim == 0 || inner == 0) return MNI_B200_OK;
    if (!p0 || !p1 || !p2) return fail(MNI_B200_ERR_ARG, "null pointer");
    if (outer > 0x7fffffffLL || inner > 0x7fffffffLL || dim > (INT64_MAX / outer) / inner ||
        (inner > 1 && outer * inner / 32 >= 0x7fffffffLL))
        return fail(MNI_B200_ERR_TOO_LARGE, "softmax extent too large");
    return MNI_B200_OK;
}

int mni_b200_softmax_fwd(const float *x, float *out, int64_t outer, int64_t dim_size, int64_t inner, void *stream) {
    int rc = softmax_args(x, out, out, outer, dim_size, inner);
    if (rc || outer * dim_size * inner == 0) return rc;
    DeviceState *st = nullptr;
    rc = device_state(&st);
    if (rc) return rc;
    return launch_softmax_fwd(x, out, outer, dim_size, inner, static_cast<cudaStream_t>(stream));
}

int mni_b200_softmax_bwd(const float *grad, const float *out, float *dx, int64_t outer, int64_t dim_size,
                         int64_t inner, void *stream) {
    int rc = softmax_args(grad, out, dx, outer, dim_size, inner);
    if (rc || outer * dim_size * inner == 0) return rc;
    DeviceState *st = nullptr;
    rc = device_state(&st);
    if (rc) return rc;
    return launch_softmax_bwd(grad, out, dx, outer, dim_size, inner, static_cast<cudaStream_t>(stream));
}

int mni_b200_grad_sumsq(const float *grad, int64_t n, double *sumsq, uint32_t flags, void *stream) {
    if (n < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (!sumsq) return fail(MNI_B200_ERR_ARG, "sumsq is null");
    if (n > 0 && !grad) return fail(MNI_B200_ERR_ARG, "grad is null");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    return launch_sumsq_list(1, &grad, &n, sumsq, (flags & MNI_B200_ACCUMULATE_C) != 0, nullptr, 0, st->sm_count,
                             static_cast<cudaStream_t>(stream));
}

// bias corrections of ops/optimizer.rs:26-27: 1 - beta.powi(step) in f32
static AdamWArgs adamw_args(float lr, float beta1, float beta2, float eps, float weight_decay, uint32_t step,
                            const double *sumsq, float max_norm, int write_clipped_grad) {
    return AdamWArgs{lr, beta1, beta2, eps, 1.0f - lr * weight_decay, 1.0f - powi_f32(beta1, step),
                     1.0f - powi_f32(beta2, step), sumsq, max_norm, write_clipped_grad ? 1 : 0};
}

int mni_b200_adamw_step(float *param, float *m, float *v, float *grad, int64_t n, float lr, float beta1, float beta2,
                        float eps, float weight_decay, uint32_t step, const double *grad_sumsq, float max_grad_norm,
                        int write_clipped_grad, void *stream) {
    if (n < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
    if (n == 0) return MNI_B200_OK;
    if (!param || !m || !v || !grad) return fail(MNI_B200_ERR_ARG, "null pointer");
    if (step == 0) return fail(MNI_B200_ERR_ARG, "step counts from 1");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    return launch_adamw_list(adamw_args(lr, beta1, beta2, eps, weight_decay, step, grad_sumsq, max_grad_norm, write_clipped_grad),
                             1, &param, &m, &v, &grad, &n, false, static_cast<cudaStream_t>(stream));
}

int mni_b200_grad_norm_sq(int64_t count, const float *const *grads, const int64_t *n, double *sumsq, void *stream) {
    if (count < 0) return fail(MNI_B200_ERR_ARG, "negative count");
    if (!sumsq || (count > 0 && (!grads || !n))) return fail(MNI_B200_ERR_ARG, "null pointer");
    for (int64_t i = 0; i < count; ++i) {
        if (n[i] < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
        if (n[i] > 0 && !grads[i]) return fail(MNI_B200_ERR_ARG, "grad is null");
    }
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    return launch_sumsq_list(count, grads, n, sumsq, false, nullptr, 0, st->sm_count, static_cast<cudaStream_t>(stream));
}

int mni_b200_clip_and_step(int64_t count, float *const *params, float *const *ms, float *const *vs, float *const *grads,
                           const int64_t *n, float lr, float beta1, float beta2, float eps, float weight_decay,
                           uint32_t step, float max_grad_norm, float *norm, void *stream) {
    if (count < 0) return fail(MNI_B200_ERR_ARG, "negative count");
    if (count > 0 && (!params || !ms || !vs || !grads || !n)) return fail(MNI_B200_ERR_ARG, "null pointer");
    for (int64_t i = 0; i < count; ++i) {
        if (n[i] < 0) return fail(MNI_B200_ERR_ARG, "negative extent");
        if (n[i] > 0 && (!params[i] || !ms[i] || !vs[i] || !grads[i])) return fail(MNI_B200_ERR_ARG, "null pointer");
    }
    if (step == 0) return fail(MNI_B200_ERR_ARG, "step counts from 1");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    cudaStream_t const s = static_cast<cudaStream_t>(stream);
    if (norm && stream_is_capturing(s))
        return fail(MNI_B200_ERR_ARG, "the norm cannot be read while the stream is capturing: pass no norm");
    double *sumsq = norm_sumsq_ptr();
    if (!sumsq) return fail(MNI_B200_ERR_CUDA, "norm accumulator unavailable");
    NormSlotLease lease;
    if (norm) {
        rc = lease.take();
        if (rc) return rc;
    }
    {
        std::lock_guard<std::mutex> lock(st->mu);      // the two launches of a call stay together
        rc = launch_sumsq_list(count, grads, n, sumsq, false, lease.slot, lease.seq, st->sm_count, s);
        if (rc == MNI_B200_OK)
            rc = launch_adamw_list(adamw_args(lr, beta1, beta2, eps, weight_decay, step, sumsq, max_grad_norm, 1), count,
                                   params, ms, vs, grads, n, true, s);
    }
    if (!norm) return rc;
    // The norm arrives while the step still runs: the host waits for it alone, not for the stream.
    const int waited = lease.wait(s);
    if (rc || waited) return rc ? rc : waited;
    *norm = sqrtf(static_cast<float>(lease.slot->sumsq));
    return MNI_B200_OK;
}

int mni_b200_contiguous(const mni_b200_view *src, float *dst, void *stream) {
    int rc = check_view(src, "src", 1);
    if (rc) return rc;
    if (prod(src->shape, src->ndim) == 0) return MNI_B200_OK;
    if (!dst) return fail(MNI_B200_ERR_ARG, "dst is null");
    DeviceState *st = nullptr;
    rc = device_state(&st);
    if (rc) return rc;
    const GatherView job{src, dst, src->shape[src->ndim - 1]};
    return launch_gather(&job, 1, static_cast<cudaStream_t>(stream));
}

int mni_b200_sm_reserve(int sms) {
    if (sms < 0) return fail(MNI_B200_ERR_ARG, "negative SM count");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(st->mu);
    st->sm_reserve = std::min(sms, std::max(0, st->sm_count - 8));
    return MNI_B200_OK;
}

int mni_b200_workspace_set(void *ptr, size_t bytes) {
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(st->mu);
    if (!ptr || bytes == 0) { st->user_ws = nullptr; st->user_bytes = 0; return MNI_B200_OK; }
    if ((reinterpret_cast<uintptr_t>(ptr) & 255) != 0) return fail(MNI_B200_ERR_ARG, "scratch must be 256-byte aligned");
    st->user_ws = static_cast<uint8_t *>(ptr);
    st->user_bytes = bytes;
    return MNI_B200_OK;
}

int mni_b200_workspace_query(const mni_b200_view *a, const mni_b200_view *b, uint32_t flags, size_t *bytes) {
    if (!bytes) return fail(MNI_B200_ERR_ARG, "bytes is null");
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    Shapes s;
    rc = analyse(a, b, s);
    if (rc) return rc;
    // The forward output's gradient, broadcast batch + [M, N], in the forms that bound what a real one can need: contiguous
    // (read in place, column sums included), the same with M and N exchanged in memory (read in place, but gathered for the
    // column sums), either on a 16-byte boundary or off it (gathered by products of f32 operands, which counts where these
    // are compared with 16-bit planes), and a view no descriptor and no plane covers (neither matrix dim has unit stride),
    // which is gathered into scratch once for each of its three uses.
    mni_b200_view dc{};
    dc.ptr = reinterpret_cast<const float *>(static_cast<uintptr_t>(256));
    dc.ndim = s.out_nb + 2;
    for (int i = 0; i < s.out_nb; ++i) dc.shape[i] = s.out_batch[i];
    dc.shape[s.out_nb] = s.M; dc.shape[s.out_nb + 1] = s.N;
    int64_t acc = 1;
    for (int d = dc.ndim - 1; d >= 0; --d) { dc.stride[d] = acc; acc *= dc.shape[d]; }
    mni_b200_view dc_strided = dc, dc_exchanged = dc;
    for (int d = 0; d < dc.ndim; ++d) dc_strided.stride[d] = dc.stride[d] * 2;
    dc_exchanged.stride[s.out_nb] = 1;
    dc_exchanged.stride[s.out_nb + 1] = s.M;
    mni_b200_view dc_off = dc, dc_exchanged_off = dc_exchanged;
    dc_off.ptr = dc_exchanged_off.ptr = dc.ptr + 1;
    size_t need = 0;
    auto dry = [&](auto body) -> int {             // eager and captured calls are planned differently
        for (const bool capturing : {false, true}) {
            Call c;
            c.st = st; c.arena.dry = true; c.stream = nullptr; c.flags = flags;
            c.capturing = capturing;
            const int r = body(c);
            if (r) return r;
            need = std::max(need, c.arena.used);
        }
        return MNI_B200_OK;
    };
    // Outputs on a 16-byte boundary and off it take different plans, and so do calls for both gradients, which may run
    // side by side on half of the SMs each, and calls for one of them.
    for (const uintptr_t at : {uintptr_t{256}, uintptr_t{260}}) {
        float *out = reinterpret_cast<float *>(at);
        rc = dry([&](Call &c) { return fwd_body(c, a, b, out, nullptr); });
        if (rc) return rc;
        for (const mni_b200_view *grad : {&dc, &dc_off, &dc_exchanged, &dc_exchanged_off, &dc_strided})
            for (int want = 1; want < 8; ++want) {
                rc = dry([&](Call &c) {
                    return bwd_body(c, a, b, grad, (want & 1) ? out : nullptr, (want & 2) ? out : nullptr, (want & 4) ? out : nullptr);
                });
                if (rc) return rc;
            }
        // bias + GELU forward without a `pre` output: when the epilogue cannot be fused the product needs a temporary
        rc = dry([&](Call &c) { return fwd_gelu_body(c, a, b, out, nullptr, out); });
        if (rc) return rc;
    }
    // the pointwise entry points on the forward output: column-sum partials
    const int64_t rows = s.batch * s.M;
    need = std::max(need, (colsum_partial_bytes(std::max<int64_t>(rows, 1), std::max<int64_t>(s.N, 1), st->sm_count) + 255) &
                              ~static_cast<size_t>(255));
    *bytes = need;
    return MNI_B200_OK;
}

int mni_b200_plan_describe(const mni_b200_view *a, const mni_b200_view *b, int backward, uint32_t flags, int sm_count,
                           char *out, size_t out_len) {
    if (!out || out_len == 0) return fail(MNI_B200_ERR_ARG, "out is null or empty");
    if (sm_count < 8 || sm_count > 4096) return fail(MNI_B200_ERR_ARG, "sm_count %d out of range", sm_count);
    out[0] = 0;
    EnvScope env;
    Shapes s;
    int rc = analyse(a, b, s);
    if (rc) return rc;
    // A stand-in for the device: the plans depend on its SM count only.
    DeviceState st;
    st.sm_count = sm_count;
    std::string log;
    Call c;
    c.st = &st; c.arena.dry = true; c.stream = nullptr; c.flags = flags; c.plan_log = &log;
    float *fake = reinterpret_cast<float *>(static_cast<uintptr_t>(256));
    if (!backward) {
        rc = fwd_body(c, a, b, fake, nullptr);
    } else {
        // the forward output's gradient: contiguous, broadcast batch + [M, N]
        mni_b200_view dc{};
        dc.ptr = fake;
        dc.ndim = s.out_nb + 2;
        for (int i = 0; i < s.out_nb; ++i) dc.shape[i] = s.out_batch[i];
        dc.shape[s.out_nb] = s.M; dc.shape[s.out_nb + 1] = s.N;
        int64_t acc = 1;
        for (int d = dc.ndim - 1; d >= 0; --d) { dc.stride[d] = acc; acc *= dc.shape[d]; }
        rc = bwd_body(c, a, b, &dc, fake, fake, backward > 1 ? fake : nullptr);
    }
    if (rc) return rc;
    if (log.size() + 1 > out_len)
        return fail(MNI_B200_ERR_ARG, "the description needs %zu bytes, %zu given", log.size() + 1, out_len);
    memcpy(out, log.c_str(), log.size() + 1);
    return MNI_B200_OK;
}

int mni_b200_device_status(void *stream, uint32_t *detail) {
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    MNI_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    unsigned int word = 0;
    MNI_CUDA(cudaMemcpy(&word, st->err_word, sizeof(word), cudaMemcpyDeviceToHost));
    if (detail) *detail = word;
    if (word != 0) {
        MNI_CUDA(cudaMemset(st->err_word, 0, sizeof(word)));
        return fail(MNI_B200_ERR_TIMEOUT, "a kernel gave up on a bounded wait (code 0x%x: role %u, slot %u)", word,
                    word >> 8, word & 0xffu);
    }
    return MNI_B200_OK;
}

int mni_b200_role_wait_cycles(uint64_t out[8], int reset) {
    if (!out) return fail(MNI_B200_ERR_ARG, "out is null");
    return read_role_waits(out, reset);
}

int mni_b200_release(void) {
    DeviceState *st = nullptr;
    int rc = device_state(&st);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(st->mu);
    st->refused = SIZE_MAX;
    if (st->ws || !st->retired.empty()) MNI_CUDA(cudaDeviceSynchronize());
    if (st->ws) {
        MNI_CUDA(cudaFree(st->ws));
        st->ws = nullptr;
        st->ws_bytes = 0;
        st->ws_recorded = false;
    }
    while (!st->retired.empty()) {
        MNI_CUDA(cudaFree(st->retired.back()));
        st->retired.pop_back();
    }
    return MNI_B200_OK;
}

}  // extern "C"
