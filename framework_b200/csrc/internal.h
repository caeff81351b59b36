// Internal interfaces between the C-ABI host logic (api.cu) and the kernel
// launchers.  Nothing here is exported.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>
#include <functional>
#include <string>

#include "mni_b200.h"

namespace mni {

// ---------------------------------------------------------------------------
// programmatic dependent launch
// ---------------------------------------------------------------------------
// Short kernels that follow one another in a stream (GEMM -> split-K finish -> GEMM, the three skinny
// products of a step) are launched with programmatic stream serialization: the next grid may be scheduled,
// and run its set-up, while its predecessor still runs; before it touches global memory it executes
// griddepcontrol.wait, which returns once the predecessor has completed and its writes are visible.
// MNI_B200_PDL=0 turns the attribute off (the device-side instructions are then no-ops).
bool pdl_enabled();
#ifdef __CUDACC__
__device__ __forceinline__ void grid_dependency_trigger() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(bool dependent, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = dependent && pdl_enabled() ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args) {
    return launch_dependent(true, kernel, grid, block, smem, stream, static_cast<Args &&>(args)...);
}
#endif

// Division by a launch-time constant as a multiply-high and a shift (exact for 0 <= n < 2^31): every role
// decodes every tile it visits, and with short contractions a handful of hardware divisions per tile showed
// up as 1 250 cycles of a 3 000-cycle main loop.  mul = ceil(2^(31 + ceil(log2 d)) / d), shr = ceil(log2 d) - 1.
struct FastDiv {
    uint32_t mul, shr, d;
};
inline FastDiv make_fastdiv(long long d_in) {
    FastDiv f;
    const uint32_t d = static_cast<uint32_t>(d_in < 1 ? 1 : d_in);
    f.d = d;
    if (d == 1) { f.mul = 0; f.shr = 0; return f; }
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;
    const uint32_t p = 31 + l;
    f.mul = static_cast<uint32_t>(((1ull << p) + d - 1) / d);
    f.shr = p - 32;
    return f;
}
#ifdef __CUDACC__
__device__ __forceinline__ int fd_div(int n, const FastDiv &f) {
    return f.d == 1 ? n : static_cast<int>(__umulhi(static_cast<uint32_t>(n), f.mul) >> f.shr);
}
#endif

// ---------------------------------------------------------------------------
// error plumbing
// ---------------------------------------------------------------------------
int fail(int status, const char *fmt, ...);          // records the thread-local message, returns status

// The MNI_B200_* switches.  A call consults some forty of them (the planner runs once to size the scratch and once to
// launch), and getenv walks the whole environment each time -- 3 of the 6 us a small product's call spent on the
// host.  An entry point opens an EnvScope, which walks the environment once; env_value then looks among the
// switches found, normally none.  Outside a scope env_value reads the environment itself.
struct EnvScope {
    EnvScope();
    ~EnvScope();
    EnvScope(const EnvScope &) = delete;
    EnvScope &operator=(const EnvScope &) = delete;
};
const char *env_value(const char *name);              // value, or nullptr if unset or empty
int env_int(const char *name, int dflt);
int device_sm_count();                                // SM count of the current device (cached per device)
extern std::atomic<uint64_t> g_launches;              // kernels launched by this library

#define MNI_CUDA(call)                                                                   \
    do {                                                                                 \
        cudaError_t e__ = (call);                                                        \
        if (e__ != cudaSuccess)                                                          \
            return ::mni::fail(MNI_B200_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e__)); \
    } while (0)

#define MNI_LAUNCH_CHECK(name)                                                           \
    do {                                                                                 \
        ::mni::g_launches.fetch_add(1, std::memory_order_relaxed);                       \
        cudaError_t e__ = cudaGetLastError();                                            \
        if (e__ != cudaSuccess)                                                          \
            return ::mni::fail(MNI_B200_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e__)); \
    } while (0)

// ---------------------------------------------------------------------------
// One GEMM operand as the tensor-core kernel reads it through a TMA descriptor.
// "rows" is the operand's non-contraction extent (M for A, N for B), "kdim" the
// contraction extent of one batch.  Exactly one of the two matrix dims has unit
// stride: k_major says which.
// ---------------------------------------------------------------------------
struct Operand {
    const float *ptr = nullptr;
    bool k_major = true;
    int64_t rows = 0, kdim = 0;
    int64_t ld = 0;                // element stride of the non-unit matrix dim
    int64_t bshape[3] = {1, 1, 1}; // operand batch dims, outermost first (front-padded with 1)
    int64_t bstride[3] = {0, 0, 0};
    int64_t batch = 1;             // product of bshape
};

// An operand in 16-bit planes (half.cu), each [batch][rows or k][pitch], and the exponent its values were multiplied by.
struct HalfOperand {
    const void *ptr = nullptr;
    bool k_major = true;
    int64_t rows = 0, kdim = 0, pitch = 0;
    int64_t matrix = 0, plane = 0;   // elements of one matrix, of one plane
    int64_t batch = 1;
    int planes = 3;                  // that there is room for
    const int *exp = nullptr;
};
// lo = (x - hi) * 2^kHalfLoShift: the whole range of f16 serves the part below hi's last bit
constexpr int kHalfLoShift = 12;
// f16 planes: exponents lie within this either way.
constexpr int kHalfMaxExp = 60;
// The exponent of bf16 planes, from that of f16 ones.  Numbers so small that their parts would run into bf16's smallest are
// scaled, unless the operand holds some that are not (huge); scaled ones stay below 1, so that no product overflows by it.
__host__ __device__ inline int half_wide_exponent(int e, bool huge) { return e == kHalfMaxExp && !huge ? 24 : 0; }

struct GemmProblem {
    Operand A, B;                  // C[M,N] = sum_k A[m,k] * B[n,k]
    int64_t M = 0, N = 0, K = 0;
    int64_t batch = 1;             // output batches
    int64_t fold = 1;              // batches summed inside the contraction (weight-gradient reduce)
    float *C = nullptr;
    int64_t ldc = 0, c_bstride = 0;
    const float *bias = nullptr;   // per output column, may be null
    bool accumulate = false;       // C += ...
    bool fast_tf32 = false;        // one TF32 pass instead of the 3-pass split
    int force_splits = 0;          // tests
    bool beside = false;           // another product runs on the SMs that this one is not planned for
    bool exchanged = false;        // the kernel's view of a product whose operands it exchanges: it computes C^T
    // Two products of one call that do not depend on each other (grad_a and grad_b) are launched back to back on
    // one stream as a pair: the first (1) lets its dependent start only after its own wait for earlier work has
    // returned, the second (2) skips that wait, runs beside the first -- on free SMs, or on the SMs its tail
    // leaves -- and waits for it just before it ends, so stream order holds for everything after the pair.
    int dep_mode = 0;
    int flag_bank = 0;             // 1 for launches on the library's side stream: their own set of balanced-tail flags
    // Optional second output D = gelu(C + bias) written by the same epilogue (C itself is skipped if null).
    float *D = nullptr;
    // The operands in 16-bit planes (A and B are not read then) and the status word of the launch that made them.
    const HalfOperand *ha = nullptr, *hb = nullptr;
    const unsigned int *half_status = nullptr;
};

// Bytes of split-K partial storage launch_gemm_tc would use for this problem (0 if none).
size_t gemm_tc_partial_bytes(const GemmProblem &p, int sm_count);

// Tensor-core path: TMA -> smem -> (hi/lo split) -> tcgen05.mma -> TMEM -> global.
// `partial` must hold gemm_tc_partial_bytes() bytes when that is non-zero.
// `defer` != null: a finish kernel (of a split contraction or a split tail) is not launched but left there; calling it
// launches it.  dep_mode 1 / 2: first / second of two finishes that do not depend on each other, launched back to back.
using GemmFinish = std::function<int(int dep_mode, cudaStream_t stream)>;
int launch_gemm_tc(const GemmProblem &p, float *partial, uint32_t *err_word, int sm_count,
                   cudaStream_t stream, GemmFinish *defer = nullptr);
// Whether the problem is computed by CTA pairs.
bool gemm_tc_uses_pairs(const GemmProblem &p, int sm_count);
// The plan's cost model for this problem in microseconds (0: the model does not cover it).
double gemm_tc_estimate_us(const GemmProblem &p, int sm_count);
// Microseconds of a product from f32 operands.
double gemm_estimate_us(const GemmProblem &p, int sm_count);
// One or two independent products from 16-bit planes (GemmProblem::ha, hb), in one launch.  partial[i] must hold bytes[i].
int launch_gemm_halves(const GemmProblem *p, int count, float *const *partial, uint32_t *err_word, int sm_count, cudaStream_t stream);
void gemm_halves_partial_bytes(const GemmProblem *p, int count, int sm_count, size_t *bytes);
double gemm_halves_estimate_us(const GemmProblem *p, int count, int sm_count);     // without the pass that makes the planes
void gemm_halves_describe(const GemmProblem *p, int count, int sm_count, std::string *lines);
// One line of text naming the kernel variant, tiling, split and grid launch_gemm_tc would use for this problem
// on a device with `sm_count` SMs.  Pure host arithmetic: touches no device.
std::string gemm_tc_describe(const GemmProblem &p, int sm_count);
// True if the fused second output (GemmProblem::D) can be produced for this problem: no split-K and a
// 16-byte aligned row pitch.  Otherwise the caller runs the GEMM and the pointwise kernel separately.
bool gemm_tc_can_fuse_activation(const GemmProblem &p, int sm_count);

// Diagnostics: copies the 8 role wait counters of the current device (collected only while
// MNI_B200_ROLE_WAITS=1 is set in the environment) and optionally clears them.
int read_role_waits(uint64_t out[8], int reset);

// Skinny path (few output rows, HBM-bound): CUDA-core fp32 FMA kernels.
//   y[M,N] = x[M,K] . W[K,N]          (W row-major, ldw)           M <= 16
int64_t skinny_fwd_row_limit(int64_t N);
bool skinny_fwd_supported(int64_t M, int64_t N, int64_t K);
size_t skinny_fwd_partial_bytes(int64_t M, int64_t N, int64_t K, int sm_count);
int launch_skinny_fwd(const float *x, int64_t ldx, const float *W, int64_t ldw, float *y, int64_t ldy,
                      const float *bias, bool accumulate, int64_t M, int64_t N, int64_t K,
                      float *partial, int sm_count, cudaStream_t stream);
//   dx[M,K] = dy[M,N] . W[K,N]^T                                    M <= 8
bool skinny_dx_supported(const float *dy, int64_t lddy, const float *W, int64_t ldw, int64_t M, int64_t N);
//   (dependent: as a programmatic dependent launch -- not beside a product on another stream, whose blocks would find
//   the waiting ones of this kernel in their places)
int launch_skinny_dx(const float *dy, int64_t lddy, const float *W, int64_t ldw, float *dx, int64_t lddx,
                     bool accumulate, int64_t M, int64_t N, int64_t K, bool dependent, cudaStream_t stream);
//   dW[K,N] = x[M,K]^T . dy[M,N]                                     M <= 16
int launch_skinny_dw(const float *x, int64_t ldx, const float *dy, int64_t lddy, float *dW, int64_t lddw,
                     bool accumulate, int64_t M, int64_t N, int64_t K, cudaStream_t stream);

// A few rows (M <= 16) in the split TF32 arithmetic of the tensor path, any alignment of the weight's rows (rows.cu).
// outs / total: outputs per row and length of the contraction (forward: N, K; dx: K, N).
bool rows_supported(int64_t M, int64_t outs, int64_t total, int sm_count);
using RowsLaunch = int(const float *x, int64_t ldx, const float *W, int64_t ldw, float *out, int64_t ldout, const float *bias,
                       bool accumulate, int64_t M, int64_t N, int64_t K, int sm_count, cudaStream_t stream);
RowsLaunch launch_rows_fwd, launch_rows_dx;            // W as stored [K, N]
RowsLaunch launch_rows_bt_fwd, launch_rows_bt_dx;      // W stored [N, K], seen through a transposing view

// Products too small for the tensor path, all of a call's in one launch (tiny.cu):
//   c[m, n] = sum_k a[m, k] . b[k, n] (+ bias) (+ c), each operand with a unit stride in one of its dims
// act != null (in the first of a call's products, and then in all): c (may be null) = the sum alone, act = gelu(sum + bias)
struct TinyProduct {
    const float *a, *b;
    float *c;
    const float *bias;
    int M, N, K, accumulate;
    long long a_m, a_k, b_k, b_n, ldc;
    float *act = nullptr;
};
//   out[j] (+)= sum_r src[r, j]
struct TinyColumns {
    const float *src;
    float *out;
    long long ld;
    int rows, n, accumulate;
};
constexpr int kMaxTiny = 2;
int launch_tiny(const TinyProduct *products, int count, const TinyColumns *columns, cudaStream_t stream);

// Pointwise / reduction helpers.
int launch_add_bias(const float *y, const float *bias, float *out, int64_t rows, int64_t n,
                    cudaStream_t stream);
size_t colsum_partial_bytes(int64_t rows, int64_t n, int sm_count);
// out = column sums of dy[rows, n] (row pitch ld); copy != null also receives dy (pitch n) in the same pass.  ticket_bank: 1 for
// calls whose partial sums are not in the library's scratch
int launch_colsum(const float *dy, int64_t ld, float *copy, float *out, int64_t rows, int64_t n, bool accumulate,
                  float *partial, int sm_count, cudaStream_t stream, int ticket_bank = 0);
int launch_copy(const float *src, float *dst, int64_t n, cudaStream_t stream);
int launch_softmax_fwd(const float *x, float *out, int64_t outer, int64_t dim, int64_t inner, cudaStream_t stream);
int launch_softmax_bwd(const float *dy, const float *out, float *dx, int64_t outer, int64_t dim, int64_t inner,
                       cudaStream_t stream);
// AdamW over a list of tensors, and the f64 sum of squares of a list of gradients (optimizer.cu).
struct AdamWArgs {
    float lr, beta1, beta2, eps, decay, bc1, bc2;
    const double *sumsq;           // squared gradient norm on the device, or null
    float max_norm;
    int write_grad;
};
struct NormSlot {                  // in pinned host memory: the squared norm, then the sequence number of the call
    double sumsq;
    unsigned seq;
};
double *norm_sumsq_ptr();          // device address of clip_and_step's squared norm
int launch_adamw_list(const AdamWArgs &a, int64_t count, float *const *param, float *const *m, float *const *v,
                      float *const *grad, const int64_t *n, bool dependent, cudaStream_t stream);
int launch_sumsq_list(int64_t count, const float *const *grad, const int64_t *n, double *out, bool accumulate,
                      NormSlot *slot, unsigned seq, int sm_count, cudaStream_t stream);
// out = gelu_tanh(x + bias[col]);  dx = grad * gelu'(x + bias), dbias = column sums of dx (partial: colsum_partial_bytes)
int launch_bias_gelu(const float *x, const float *bias, float *out, int64_t rows, int64_t n, cudaStream_t stream);
int launch_bias_gelu_bwd(const float *grad, const float *x, const float *bias, float *dx, float *dbias,
                         int64_t rows, int64_t n, bool accumulate, float *partial, int sm_count,
                         cudaStream_t stream);
// dst[row-major, ld_dst on the last dim] = gather of a strided view; several views of a call in one launch (gather.cu)
struct GatherView {
    const mni_b200_view *src;
    float *dst;
    int64_t ld_dst;
};
constexpr int kMaxGathers = 3;
int launch_gather(const GatherView *views, int count, cudaStream_t stream);
// Matrices to be made into 16-bit planes (half.cu): `batch` of them, rows x cols, unit stride along cols.
struct HalfView {
    const float *src;
    int64_t bshape[3], bstride[3], batch;
    int64_t rows, cols, ld;
    void *dst;                     // the planes, rows of `pitch` elements (a multiple of 64)
    int64_t pitch, matrix, plane;
    int *exp;                      // on the device: the exponent the values were multiplied by
};
constexpr int kMaxHalves = 3;
int half_blocks(const HalfView *views, int count, int sm_count);      // blocks of the launches
// status: a word per block, and one for all of them behind those (bit 0: the planes are bf16, bit 1: see half_wide_exponent)
// Column sums of the first view's rows, for the bias gradient (out null: none).
struct HalfColumns {
    float *partial = nullptr, *out = nullptr;
    int accumulate = 0;
};
size_t half_columns_bytes(const HalfView &first, int blocks);
// planes: 3, for products in full precision (f16 hi and lo, or three bf16), or 2, for single-pass ones (f16 hi, or two bf16)
int launch_split_half(const HalfView *views, int count, int planes, unsigned int *status, int blocks, const HalfColumns &sums,
                      cudaStream_t stream);
// device-side utils::unbroadcast: out[orig] (+)= sum over broadcast dims of grad[gshape]
int launch_unbroadcast(const float *grad, const int64_t *gshape, int gnd, const int64_t *oshape, int ond,
                       float *out, bool accumulate, cudaStream_t stream);

}  // namespace mni
