// Tensor-core GEMM for sm_100a: C[M,N] = sum_k A[m,k] * B[n,k] on f32 storage.
//
// Data path of one CTA (persistent over output tiles, one CTA per SM; 2 + NS + 8 warps):
//
//   warp 0      TMA producer: cp.async.bulk.tensor (5-D maps: matrix dims + batch dims) brings
//               a 128 x BK tile of A and a BN x BK tile of B into a swizzled shared-memory
//               stage.  K-major and MN-major operands differ only in the tensor map and the
//               box list, so transposed / permuted operands are read in place -- no transposed
//               copy is ever written.
//   warps 2..   split (NS = 8 warps; 4 idle relays in single-pass mode): for every f32 x of the
//               landed stage, lo = x - trunc_tf32(x) (exact in f32) is written to a sibling buffer
//               of identical layout (the split is position independent, so it needs no knowledge
//               of the swizzle).  The landed tile itself serves as hi: the tensor core ignores the
//               low 13 mantissa bits of a TF32 operand (tests/test_matmul_gpu.py pins that).
//               Narrow tiles (BN <= 128, lone CTA) instead move A into tensor memory: each thread
//               reads 16 k-values of its row and stores hi and lo with tcgen05.st; only B keeps a
//               lo copy in shared memory.  For long contractions the eight warps take alternate
//               k-blocks as two groups of four (SG = 2), so two k-blocks are in flight.  When the
//               tile is wider than the output, MMAs, B box and lo copy cover only the live columns.
//   warp 1      issues tcgen05.mma.kind::tf32 per 8-deep k-step: lo*hi, hi*lo, hi*hi into one f32
//               accumulator in TMEM ("3xTF32"); one MMA on the raw tile in single-pass mode.  The
//               warp runs its loop uniformly and predicates the issue with elect.sync, and it reads
//               the next stage's barrier before queueing this stage's MMAs.
//   last 8      epilogue, two warps per TMEM lane quarter, half of the tile's columns each:
//               tcgen05.ld of the accumulator (double buffered in TMEM, so it overlaps the next
//               tile's main loop), bias add in registers, 128B-swizzled staging patch, TMA store
//               (or TMA reduce-add for C += ...) of 32 x 32 boxes; the tensor map clips the M / N
//               tails.  Split-K partials go through the same path into scratch.  Outputs whose row
//               pitch is not a multiple of 16 bytes take a plain-store fallback.
//
// Large products take their operands as 16-bit planes instead, which half.cu makes of them beforehand (kHalfThree, kHalfOne): the
// f16 pipe has the eleven bits of TF32 at twice the rate.  Nothing is split here then; the split warps only relay "landed".
//   kHalfThree  per k-block of 64: hi*hi into one accumulator, lo*hi and hi*lo (scaled by 2^12) into another, both of them all of
//               tensor memory.  The epilogue takes both into its registers and the next unit begins; the large terms' chain is a
//               third as long as in 3xTF32, and its rounding a sixth (1.24e-6 -> 3.5e-7 at K = 512, 7.6e-6 -> 1.25e-6 at 2048
//               to 3072), so a piece may be 4096 long.  Bound by the power cap in a loop, by L2 (16 KB a CTA and 16 elements) at
//               full clocks.  8192^3: 24.4 cycles per element of a tile for the pipe's 24, 4.0 -> 2.5 ms a product with the pass
//               over the operands, in a loop; as one accumulator with hi staged a second time, 33 cycles (L2).
//   kHalfOne    hi*hi alone, accumulators double-buffered as in single-pass TF32: 9.4 cycles for the pipe's 8 (L2: 8 KB a CTA and
//               16 elements), 1.8 -> 0.96 ms.
// Operands whose range f16 does not hold come as three (two) bf16 planes through the same stages.
//
// CG = 2: two CTAs of a cluster share a 256 x BN tile (cta_group::2 MMAs issued by the leader).
// Work is dealt out as whole tiles, round-robin over the CTAs (pairs).  The tiles of a badly ragged wave are cut into
// several units each, whose partial tiles go to scratch and are added by tail_finish_kernel (cut_tail has the rule).  On
// request (MNI_B200_STREAMK=1) its k-blocks are dealt out in equal ranges instead, and a tile shared by several CTAs is summed in
// slot order by whichever of them finishes last (tickets and flags in global memory, bounded waits).
//
// The tensor core's f32 accumulate rounds toward zero (measured: 2.35e-9 * K relative per chain, three
// chains' worth in 3xTF32), so a long contraction is not summed in one accumulator: a unit is handed
// out in pieces of at most KParams::chunk_iters k-blocks (an eighth more stays whole), each piece gets a fresh accumulator, and
// the epilogue adds the pieces up in its registers (256-wide pairs) or adds the later ones to the output with ordered TMA
// reduce-adds; the order is fixed either way: reproducible.
//
// Every wait on an mbarrier or flag is bounded: after KParams::wait_cycles clock cycles (~2 s unless a
// test shortens it) the waiter records a code in a global error word, raises a CTA-wide abort flag and
// all roles drain to the common exit, where TMEM is released.  Nothing traps.
#include "activation.h"
#include "internal.h"

#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <unordered_map>

namespace mni {

namespace {

constexpr int BM = 128;
constexpr int kMaxStages = 8;
constexpr int kSkMaxShare = 6;                             // balanced tail: most units that may share one tile
constexpr int kEpiWarps = 8;                                // two per TMEM lane quarter, half of the columns each
constexpr int kEpiBufBytes = 32 * 128;                     // one 32 x 32 f32 patch
constexpr int kBarBytes = (3 * kMaxStages + 4) * 8 + 16;
constexpr long long kWaitCycles = 4000000000LL;            // default limit of every device-side wait: ~2 s at 2 GHz

enum OperandMode { kKMajor = 0, kMnMultiBox = 1, kMnSingleBox = 2 };
enum TailMode { kWholeTiles = 0, kBalanced = 1, kCutTiles = 2, kRunningSum = 3 };
// How a product is computed: operands as f32 (three TF32 passes, or one), or as the 16-bit halves that split_half_kernel has made
// of them (three passes, or one).
enum PassMode { kThreePass = 0, kOnePass = 1, kHalfThree = 2, kHalfOne = 3 };
enum EpilogueMode { kEpiPlainStores = 0, kEpiTmaStore = 1, kEpiTmaReduce = 2, kEpiVectorStores = 3 };

struct KParams {
    int M, N;
    int tiles_m, tiles_n, group_m;
    int batch;                 // output batches
    int kiters;                // k-blocks per folded batch
    int fold;
    int splits;
    int dep_mode;              // 0: depends on everything before it; 1 / 2: first / second of two independent products (see GemmProblem)
    int chunk_iters;           // longest run of k-blocks summed in one tensor-memory accumulator (0 = no limit)
    int a_batch, a_d1, a_d2;   // operand flat batch count and inner dim sizes
    int b_batch, b_d1, b_d2;
    int a_mode, b_mode;        // OperandMode
    int stages;
    int epi_mode;              // EpilogueMode
    int epi_patches;           // staging patches per epilogue warp: TMA stores in flight per warp
    uint32_t idesc;
    // A tile wider than the output (lone CTA, K-major B): the B box, the lo copy and the MMAs cover only the rows
    // that exist.  b_rows_live = rows of the B tile that are loaded and split (the tile's width otherwise).
    int b_rows_live;
    uint32_t a_desc_hi, b_desc_hi;   // upper 32 bits of the smem descriptors (SBO | version | layout)
    uint32_t a_desc_lbo, b_desc_lbo; // LBO field, already shifted into the low word
    uint32_t a_kstep, b_kstep;       // descriptor address advance (16-byte units) per 8-deep k-step
    float *C;
    long long ldc, c_bstride;
    float *partial;            // split-K: [split][batch][M][partial_ld]
    long long partial_ld;      // N rounded up to a multiple of 4, so that partials always leave through TMA
    const float *bias;
    int accumulate;
    int transpose_out;         // the kernel computes C^T (operands exchanged): patches are stored transposed, bias is per row
    int act;                   // 1: also emit gelu(acc + bias) through the second output map
    int store_pre;             // act mode: write the raw product through the first map as well
    FastDiv fd_splits, fd_per_batch, fd_group_sz, fd_group_m, fd_last_gm;   // decode_unit
    FastDiv fd_a_cnt, fd_a_d1, fd_a_d2, fd_b_cnt, fd_b_d1, fd_b_d2;         // batch_coords
    unsigned int *err;
    long long wait_cycles;     // limit of every bounded wait in clock cycles (kWaitCycles unless a test shortens it)
    int withhold_at;           // test hook: the producer arms its n-th k-block (1-based) but issues no copy for it; 0 = off
    unsigned long long *prof;  // optional role wait counters (null = off)
    // Balanced tail ("stream-K"): tiles [sk_first_tile, tiles) are not dealt out whole; their k-blocks are
    // cut into one contiguous range per CTA (pair), so a ragged last wave costs its share, not a full wave.
    int sk;                    // 0 = off
    // Split tail: units below `tail_unit` are whole tiles, the rest are the last wave's tiles cut into `tail_ways` units each,
    // whose partial tiles go to scratch (through tmP) for tail_finish_kernel.  units = all of them.
    int units, tail_unit, tail_ways;
    FastDiv fd_ways;
    int sk_first_tile;         // tiles below this index are dealt out whole, round-robin
    float *sk_partial;         // two parked accumulator tiles per CTA: [cta][2][epilogue warp][chunk][8][lane] float4
    unsigned int *sk_flags;    // ready flags [cta][2][epilogue warp] (1 = parked), then tickets [tile][rank][epilogue warp]
    // 16-bit halves: what split_half_kernel left beside them
    const int *a_exp, *b_exp;              // the operands were multiplied by 2^exponent
    const unsigned int *half_status;       // bit 0: some operand's range did not fit
};

// What a launch computes: one product, or (16-bit planes) two that need nothing from each other, the units of the second dealt
// out after those of the first to the CTA pairs whose turn it is.
struct Product {
    CUtensorMap A, B, C, D, P;
    KParams p;
};
template <int N>
struct Products {
    Product s[N];
    int count;
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// Bounded wait.  Returns false if the CTA is aborting (this waiter or another gave up).
// With `timed`, `waited` accumulates the cycles spent blocked (role-level wait accounting, including
// the time the first try_wait is suspended by the hardware); without it the satisfied case costs one
// try_wait and no clock reads.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag,
                                          unsigned int *err, uint32_t code, long long &waited, bool timed,
                                          long long limit) {
    long long t0 = 0;
    if (timed) t0 = clock64();
    if (mbar_try_wait(bar, parity)) {
        if (timed) waited += clock64() - t0;
        return true;
    }
    if (!timed) t0 = clock64();
    uint32_t spins = 0;
    while (true) {
        if (mbar_try_wait(bar, parity)) {
            if (timed) waited += clock64() - t0;
            return true;
        }
        if ((++spins & 63u) == 0u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > limit) {
                *abort_flag = 1u;
                atomicCAS(err, 0u, code);
                return false;
            }
        }
    }
}
// Warp-collective form: every lane polls, the verdict is made uniform.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag,
                                               unsigned int *err, uint32_t code, long long &waited, bool timed,
                                               long long limit) {
    const bool ok = mbar_wait(bar, parity, abort_flag, err, code, waited, timed, limit);
    return __all_sync(0xffffffffu, ok);
}
// Non-blocking look at a barrier phase (try_wait may suspend the thread; this never does).
__device__ __forceinline__ uint32_t mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// True in exactly one lane of a converged warp.  The TMA and MMA issuing warps run their loops
// warp-uniformly and predicate only the issuing instruction with this: descriptors and
// coordinates then stay in uniform registers, which makes an MMA issue ~3x cheaper than from a
// single-lane branch (measured: 40 vs 120 cycles).
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .b32 rx;\n\t.reg .pred px;\n\t"
        "elect.sync rx|px, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, px;\n\t}"
        : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0,
                                            int c1, int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
        "r"(c4)
        : "memory");
}
__device__ __forceinline__ void tma_store_5d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(0), "r"(0)
                 : "memory");
}
__device__ __forceinline__ void tma_reduce_add_5d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2) {
    asm volatile(
        "cp.reduce.async.bulk.tensor.5d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
        ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(0), "r"(0)
        : "memory");
}
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                          uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %5, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// A operand from tensor memory (lanes = rows, one 32-bit column per k element), B from shared memory.
__device__ __forceinline__ void umma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
// ---- CTA-pair (cta_group::2) forms: one MMA spans two SMs; the leader CTA issues it.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on the barrier at the same shared-memory offset in CTA `cta` of the cluster.
__device__ __forceinline__ void mbar_arrive_cta(uint32_t bar, uint32_t cta) {
    asm volatile(
        "{\n\t.reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}"
        ::"r"(bar), "r"(cta)
        : "memory");
}
__device__ __forceinline__ void umma_tf32_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                               uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], da, db, %5, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                              uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Commit that arrives on the barrier at this offset in both CTAs of the pair.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(bar), "h"(static_cast<uint16_t>(3))
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
          "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
          "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
          "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct TileCoord {
    int bt, tm, tn, split, it0, it1;
    int shared;      // balanced tail: this unit is only a range of the tile's k-blocks
    int park;        // shared: which of the CTA's two parking places it uses (0 = first unit of its range)
    int tile;        // flat tile index
    int part;        // >= 0: index of this unit among the split tail's
    int chunk;       // > 0: a later piece of a unit whose contraction is summed in several accumulators (added to the output)
};

template <int TAIL>
__device__ __forceinline__ TileCoord decode_unit(const KParams &p, int unit) {
    TileCoord t;
    t.part = TAIL == kCutTiles ? unit - p.tail_unit : -1;
    int tile, ways;
    if (t.part >= 0) {
        const int q = fd_div(t.part, p.fd_ways);
        ways = p.tail_ways;
        tile = p.tail_unit + q;                    // whole tiles before the tail: unit == tile there
        t.split = t.part - q * ways;
    } else {
        ways = p.splits;
        tile = fd_div(unit, p.fd_splits);
        t.split = unit - tile * ways;
    }
    t.shared = 0;
    t.park = 0;
    t.chunk = 0;
    t.tile = tile;
    const int per_batch = p.tiles_m * p.tiles_n;
    t.bt = fd_div(tile, p.fd_per_batch);
    const int r = tile - t.bt * per_batch;
    const int group_sz = p.group_m * p.tiles_n;
    const int g = fd_div(r, p.fd_group_sz);
    const int first_m = g * p.group_m;
    const int gm = min(p.group_m, p.tiles_m - first_m);       // the last group may be shorter
    const int rin = r - g * group_sz;
    t.tn = gm == p.group_m ? fd_div(rin, p.fd_group_m) : fd_div(rin, p.fd_last_gm);
    t.tm = first_m + (rin - t.tn * gm);
    const int total = p.fold * p.kiters;
    if (ways == 1) {
        t.it0 = 0;
        t.it1 = total;
    } else {
        t.it0 = static_cast<int>(static_cast<long long>(total) * t.split / ways);
        t.it1 = static_cast<int>(static_cast<long long>(total) * (t.split + 1) / ways);
    }
    return t;
}

// The work of one CTA (pair), in the order every role walks it: whole tiles slot, slot + P, ... and then,
// with the balanced tail on, this slot's contiguous range of the tail's k-blocks, which touches at most the
// end of one tile, whole tiles, and the beginning of one tile.
struct WorkIter {
    int unit, unit_step, unit_end;     // whole units
    long long w0, w, w1;               // tail range in k-blocks, relative to the tail's first tile
    // A unit with a long contraction is handed out as consecutive pieces of at most p.chunk_iters k-blocks:
    // the tensor core's f32 accumulate truncates, so one long chain loses ~7e-9 * K of relative accuracy;
    // every piece gets a fresh accumulator and the epilogue adds it to the output (round-to-nearest adds).
    TileCoord cur;                     // the unit being handed out in pieces
    int piece_it, piece_end, piece_len, piece_no;
};
__device__ __forceinline__ long long sk_range_begin(const KParams &p, int slot, int nslots) {
    const long long total = static_cast<long long>(p.batch * p.tiles_m * p.tiles_n - p.sk_first_tile) * (p.fold * p.kiters);
    return total * slot / nslots;
}
__device__ __forceinline__ WorkIter work_begin(const KParams &p, int slot, int nslots) {
    WorkIter wi;
    wi.unit = slot;
    wi.unit_step = nslots;
    wi.unit_end = p.sk ? p.sk_first_tile : p.units;
    wi.w0 = wi.w = wi.w1 = 0;
    wi.piece_it = wi.piece_end = wi.piece_len = wi.piece_no = 0;
    if (p.sk) {
        wi.w0 = wi.w = sk_range_begin(p, slot, nslots);
        wi.w1 = sk_range_begin(p, slot + 1, nslots);
    }
    return wi;
}
// Cuts a long unit into equal pieces of at most p.chunk_iters k-blocks: `t` becomes the first piece, the iterator
// remembers the rest.
__device__ __forceinline__ void first_piece(const KParams &p, WorkIter &wi, TileCoord &t) {
    const int len = t.it1 - t.it0;
    if (p.chunk_iters > 0 && len > p.chunk_iters + (p.chunk_iters >> 3)) {
        const int pieces = (len + p.chunk_iters - 1) / p.chunk_iters;
        wi.cur = t;
        wi.piece_len = (len + pieces - 1) / pieces;
        wi.piece_end = t.it1;
        wi.piece_no = 0;
        t.it1 = t.it0 + wi.piece_len;
        wi.piece_it = t.it1;
    }
}
template <int TAIL>
__device__ __forceinline__ bool work_next(const KParams &p, WorkIter &wi, TileCoord &t) {
    if (wi.piece_it < wi.piece_end) {          // next piece of the current unit
        t = wi.cur;
        t.it0 = wi.piece_it;
        t.it1 = min(wi.piece_end, wi.piece_it + wi.piece_len);
        t.chunk = ++wi.piece_no;
        wi.piece_it = t.it1;
        return true;
    }
    if (wi.unit < wi.unit_end) {
        t = decode_unit<TAIL>(p, wi.unit);
        wi.unit += wi.unit_step;
        first_piece(p, wi, t);
        return true;
    }
    if (TAIL == kBalanced && wi.w < wi.w1) {
        const int per_tile = p.fold * p.kiters;
        const int rel = static_cast<int>(wi.w / per_tile);
        const int it0 = static_cast<int>(wi.w - static_cast<long long>(rel) * per_tile);
        const int it1 = static_cast<int>(min(static_cast<long long>(per_tile), it0 + (wi.w1 - wi.w)));
        t = decode_unit<TAIL>(p, p.sk_first_tile + rel);          // splits == 1 here: unit == tile
        t.it0 = it0;
        t.it1 = it1;
        t.shared = (it0 != 0 || it1 != per_tile) ? 1 : 0;
        t.park = wi.w == wi.w0 ? 0 : 1;
        wi.w += it1 - it0;
        // A whole tile inside a tail range is summed in pieces like any other unit; a cut tile is not (its one
        // accumulator is what gets parked or reduced), so its chain is as long as its share of the contraction.
        if (!t.shared) first_piece(p, wi, t);
        return true;
    }
    return false;
}

__device__ __forceinline__ void batch_coords(int q, int cnt, int d1, int d2, const FastDiv &fcnt, const FastDiv &fd1,
                                             const FastDiv &fd2, int &c0, int &c1, int &c2) {
    q = cnt == 1 ? 0 : q - fd_div(q, fcnt) * cnt;
    const int r = fd_div(q, fd2);
    c2 = q - r * d2;
    c0 = fd_div(r, fd1);
    c1 = r - c0 * d1;
}

// Issues the TMA copies of one operand tile.  row0 = first row of the tile, nchunk = tile rows / 32.
__device__ __forceinline__ void load_operand(int mode, uint32_t dst, const CUtensorMap *map, uint32_t bar, int k0,
                                             int row0, int nchunk, uint32_t chunk_bytes, int c0, int c1, int c2) {
    if (mode == kKMajor) {
        tma_load_5d(dst, map, bar, k0, row0, c2, c1, c0);
    } else if (mode == kMnSingleBox) {
        tma_load_5d(dst, map, bar, 0, k0, row0 >> 5, c2, c1);
    } else {
        for (int c = 0; c < nchunk; ++c) tma_load_5d(dst + c * chunk_bytes, map, bar, row0 + c * 32, k0, c2, c1, c0);
    }
}

// The same for a tile of 16-bit halves: 64 elements of the contiguous dimension wide, 128 rows.
__device__ __forceinline__ void load_half(int mode, uint32_t dst, const CUtensorMap *map, uint32_t bar, int k0, int row0, int batch,
                                          int plane) {
    if (mode == kKMajor) tma_load_5d(dst, map, bar, k0, row0, batch, plane, 0);
    else tma_load_5d(dst, map, bar, 0, k0, row0 >> 6, batch, plane);
}

// CG = 1: one CTA computes a 128 x BN tile.  CG = 2: a pair of CTAs (a 2-CTA cluster) computes a
// 256 x BN tile with cta_group::2 MMAs issued by the pair's leader; each CTA stages its own 128 rows
// of A and half (BN/2 rows) of B, so shared-memory and L2 traffic per flop drop by a third.
// TA = true (3xTF32, lone CTA, BK = 32, BN <= 128): the A operand of the MMAs comes from tensor memory.
// The split warps read each landed A row once, and store hi and lo with tcgen05.st into a TMEM slot
// of the stage (columns 2*BN + stage*64: 32 of hi, 32 of lo); no lo copy of A is written to shared
// memory and no MMA re-reads A from it, which is what bounds narrow tiles otherwise.
// TAIL: what the last wave may be.  kWholeTiles; kBalanced compiles the balanced tail's epilogue (parking / reducing
// shared tiles) in; kCutTiles the split tail's (partial tiles to scratch).  kRunningSum: whole tiles whose contraction is
// summed in several pieces, added up in the epilogue's registers instead of in memory (256-wide pairs, TMA stores, no
// activation): 8192^3 single-pass 5.97 -> 5.53 ms a step, 3xTF32 1 %; its wide epilogue costs single-piece tiles 15 %.
// Each instantiation carries only its own code and registers (2 % of a single-pass 8192^3 product otherwise).
// SG = 2 (TA only): the split warps work as two groups on alternate k-blocks (see the split role).
__host__ __device__ constexpr int gemm_threads(int ns, bool run) { return 32 * ((run ? 4 : 2) + ns + kEpiWarps); }
// Register shares of the running-sum variants, in registers per thread, out of what the launch gives each thread (96 of
// 640 threads, 128 of 512 in single-pass mode): two epilogue warpgroups, the split's and the one that issues.
template <int MODE>
struct RegShare {
    static constexpr bool kPlain = MODE == kThreePass, kOneF32 = MODE == kOnePass;
    static constexpr int kEpilogue = kPlain ? 168 : kOneF32 ? 216 : 208, kSplit = kOneF32 ? 40 : 48, kIssue = kOneF32 ? 40 : 48;
    static constexpr int kSplitGroups = kPlain ? 2 : 1, kLaunch = kPlain ? 96 : 128;
    static_assert(2 * kEpilogue + kSplitGroups * kSplit + kIssue <= (3 + kSplitGroups) * kLaunch, "more registers than the launch has");
};
// ... and of the two-accumulator variant, 168 of 384 threads at launch: two epilogue warpgroups and the one of all other roles.
constexpr int kTwoEpilogue = 224, kTwoIssue = 56, kTwoLaunch = 168;
static_assert(2 * kTwoEpilogue + kTwoIssue <= 3 * kTwoLaunch, "more registers than the launch has");
__host__ __device__ constexpr int product_slots(int mode) { return mode == kHalfThree || mode == kHalfOne ? 2 : 1; }
template <int BN, int BK, int MODE, int NS, int CG, bool TA = false, int TAIL = kWholeTiles, int SG = 1>
__global__ void __launch_bounds__(gemm_threads(NS, TAIL == kRunningSum), 1)
gemm_tc_kernel(const __grid_constant__ Products<product_slots(MODE)> g) {
    const KParams &p = g.s[0].p;                           // what every product of the launch shares is read there
    constexpr bool SK = TAIL == kBalanced, CUT = TAIL == kCutTiles;
    constexpr bool HALF = MODE == kHalfThree || MODE == kHalfOne, FAST = MODE != kThreePass;   // FAST: the split warps split nothing
    static_assert(!HALF || (BN == 256 && BK == 64 && CG == 2 && !TA && !SK), "16-bit halves are built for 256-wide pairs");
    constexpr uint32_t ELT = HALF ? 2 : 4;                 // bytes of a staged element
    constexpr int BNL = BN / CG;                           // B rows staged by this CTA
    constexpr uint32_t A_BYTES = BM * BK * ELT;
    constexpr uint32_t B_BYTES = BNL * BK * ELT;
    constexpr uint32_t RAW_BYTES = A_BYTES + B_BYTES;
    // RUN: a unit's running sum over its pieces takes 128 registers of every epilogue thread, so the warps are laid out in
    // whole warpgroups -- TMA and MMA (and two idle), split, epilogue -- that trade registers.
    // TWO: the large and the small terms of a piece in an accumulator each, all of tensor memory; the epilogue takes both into its
    // registers, whole, before anything is stored, and the next piece begins.
    constexpr bool TWO = MODE == kHalfThree, RUN = TAIL == kRunningSum || TWO;
    static_assert(!RUN || (BN == 256 && CG == 2), "running sums are built for 256-wide pairs");
    constexpr int SPLIT0 = RUN && !TWO ? 4 : 2, EPI0 = SPLIT0 + NS;   // first split and first epilogue warp
    static_assert(!TA || (!FAST && CG == 1 && BK == 32 && NS == 8 && BN <= 128), "unsupported A-from-TMEM variant");
    constexpr uint32_t STAGE_BYTES = FAST ? RAW_BYTES : (TA ? A_BYTES + 2 * B_BYTES : 2 * RAW_BYTES);
    constexpr uint32_t STAGE16 = STAGE_BYTES >> 4;
    constexpr uint32_t LO16 = (TA ? B_BYTES : RAW_BYTES) >> 4;   // lo copy relative to its raw tile, 16-byte units
    constexpr int KSTEPS = BK / (HALF ? 16 : 8);
    constexpr uint32_t TMEM_COLS = TA ? 512 : 2 * BN;      // double-buffered accumulator (+ the A slots)
    constexpr uint32_t TA_COL0 = 2 * BN;                   // first column of the A slots
    constexpr uint32_t TA_SLOT = 2 * BK;                   // hi | lo

    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                ~static_cast<uintptr_t>(1023));
    uint8_t *stage_base = smem;
    uint8_t *epi_base = smem + static_cast<size_t>(p.stages) * STAGE_BYTES;      // 1024-aligned
    uint64_t *bars = reinterpret_cast<uint64_t *>(epi_base + kEpiWarps * p.epi_patches * kEpiBufBytes);
    // bars: full[S] | xform[S] | empty[S] | acc_full[2] | acc_empty[2]
    const uint32_t bar_full = smem_u32(bars);
    const uint32_t bar_xform = bar_full + 8u * kMaxStages;
    const uint32_t bar_empty = bar_xform + 8u * kMaxStages;
    const uint32_t bar_acc_full = bar_empty + 8u * kMaxStages;
    const uint32_t bar_acc_empty = bar_acc_full + 16u;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * kMaxStages + 4);
    volatile uint32_t *abort_flag = tmem_slot + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const bool timed = p.prof != nullptr;
    const long long t_kernel0 = clock64();
    const uint32_t cta_rank = CG == 2 ? cluster_ctarank() : 0u;   // 0 = the pair's leader
    const int unit0 = static_cast<int>(blockIdx.x) / CG;           // this CTA (pair) starts at this unit ...
    const int unit_step = static_cast<int>(gridDim.x) / CG;        // ... and strides by the number of CTAs (pairs)

    // The next grid in the stream may be scheduled already -- unless it is the independent second product of
    // a pair, which skips its own wait: then it may only start once this grid's predecessors are known complete.
    if (threadIdx.x == 0 && p.dep_mode != 1) grid_dependency_trigger();
    if (warp == 0 && lane == 1) {
        // descriptor fetches overlap the barrier and TMEM set-up
        for (int prod = 0; prod < (HALF ? g.count : 1); ++prod) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&g.s[prod].A)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&g.s[prod].B)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&g.s[prod].C)) : "memory");
        }
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(bar_full + 8u * s, 1);
            mbar_init(bar_xform + 8u * s, HALF ? CG : CG * NS / SG);   // one arrival per split warp (of the k-block's group; of both CTAs for a pair)
            mbar_init(bar_empty + 8u * s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_acc_full + 8u * i, 1);
            mbar_init(bar_acc_empty + 8u * i, CG * kEpiWarps);   // one arrival per epilogue warp, of both CTAs for a pair
        }
        *abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             smem_u32(tmem_slot)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             smem_u32(tmem_slot)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CG == 2) cluster_sync_all();   // the peer's barriers exist before anyone arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Everything above overlapped the previous grid; its results are needed from here on.  The second product of
    // an independent pair needs nothing from the first: it runs beside it and waits for it only before it ends.
    if (p.dep_mode != 2) grid_dependency_wait();
    if (p.dep_mode == 1 && threadIdx.x == 0) grid_dependency_trigger();
    // HALF: wide if some operand's range did not fit f16, and the planes hold bf16 thirds, unscaled.
    bool wide = false, huge = false;
    if constexpr (HALF) {
        const unsigned int status = __ldcg(p.half_status);
        wide = (status & 1u) != 0;
        huge = (status & 2u) != 0;
    }
    // The products of the launch, as every role walks them: first_unit is this CTA pair's first unit of one.
    const int products = HALF ? g.count : 1;
    auto first_unit = [&](int prod) {
        if (prod == 0) return unit0;
        const int at = unit0 - g.s[0].p.units % unit_step;
        return at < 0 ? at + unit_step : at;
    };
    const int planes = TWO ? (wide ? 3 : 2) : (wide ? 2 : 1);     // HALF

    // The epilogue comes first: it is the branch whose register share the running-sum variants raise.
    if (warp >= EPI0) {
        // RUN: the warpgroups trade registers; the increase waits for the others' decrease
        if constexpr (RUN) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TWO ? kTwoEpilogue : RegShare<MODE>::kEpilogue));
        // ------------------------------------------------------------ epilogue
        const int quarter = warp & 3;                       // TMEM lane quarter this warp may read
        const int ew = warp - EPI0;               // 0..7: warps ew and ew+4 share a lane quarter ...
        constexpr int CHUNKS = BN / 32 / (kEpiWarps / 4);   // ... and take half of the tile's 32-column chunks each
        const int chunk_lo = (ew >> 2) * CHUNKS;
        uint8_t *my_stage = epi_base + ew * p.epi_patches * kEpiBufBytes;
        int acc_it = 0;
        int patch = 0;                                // staging buffer to use next
        int in_flight = 0;                            // bulk groups committed by lane 0 and not yet waited for
        bool ok = true;
        long long waited = 0, t_ld = 0, t_wg = 0;
        const int my_cta = static_cast<int>(blockIdx.x);                 // slot * CG + rank in the pair
        for (int prod = 0; ok && prod < products; ++prod) {
        const Product &w = g.s[HALF ? prod : 0];
        const KParams &q = HALF ? w.p : p;
        float unscale = 1.f;
        if constexpr (HALF) {
            int ea = __ldcg(q.a_exp), eb = __ldcg(q.b_exp);          // at most 60 either way
            if (wide) { ea = half_wide_exponent(ea, huge); eb = half_wide_exponent(eb, huge); }
            unscale = __uint_as_float(static_cast<uint32_t>(127 - ea - eb) << 23);
        }
        const bool use_tma = q.epi_mode == kEpiTmaStore || q.epi_mode == kEpiTmaReduce;
        const bool bias_vec = (reinterpret_cast<uintptr_t>(q.bias) & 15) == 0;
        WorkIter wi = work_begin(q, first_unit(prod), unit_step);
        TileCoord t;
        uint32_t run[RUN ? CHUNKS : 1][32];           // RUN: sum of the unit's pieces so far
        while (ok && work_next<TAIL>(q, wi, t)) {
            const int buf = TWO ? 0 : acc_it & 1;
            const uint32_t acc_phase = TWO ? acc_it & 1 : (acc_it >> 1) & 1;
            ok = mbar_wait(bar_acc_full + 8u * buf, acc_phase, abort_flag, p.err, 0x500u | buf, waited, timed, p.wait_cycles);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const bool part = CUT && t.part >= 0;            // of the split tail: a raw partial tile, always through TMA
            const bool fuse = q.splits == 1 && !part;
            const bool tma_here = use_tma || part;
            const bool later_piece = t.chunk > 0;     // a later piece of this unit's contraction: added to the earlier ones
            const bool last_piece = wi.piece_it >= wi.piece_end;
            const bool add_piece = !RUN && later_piece;   // ... through memory
            if (add_piece && tma_here) {
                // this warp's earlier stores to the same patches must have completed, not just been read
                if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                in_flight = 0;
                __syncwarp();
            }
            const int row0 = t.tm * (BM * CG) + static_cast<int>(cta_rank) * BM + quarter * 32;
            const int cbatch = fuse ? t.bt : t.split * q.batch + t.bt;
            const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(buf * BN);
            // Shared tile of the balanced tail.  Each (tile, CTA rank, epilogue warp) region has a ticket; the
            // units of the tile arrive in any order, all but the last park their accumulator (and raise a
            // ready flag), the last one adds the parked ones to its own in slot order -- the sum does not
            // depend on who came last -- and runs the usual epilogue.
            int seg_first = 0, seg_count = 1;          // slots sharing the tile: seg_first .. seg_first + seg_count - 1
            bool reducer = false;
            const int nslots = static_cast<int>(gridDim.x) / CG;
            if (SK && t.shared) {
                const long long per_tile = q.fold * q.kiters;
                const long long tile_begin = static_cast<long long>(t.tile - p.sk_first_tile) * per_tile;
                const long long tile_end = tile_begin + per_tile;
                seg_first = unit0;
                while (seg_first > 0 && sk_range_begin(p, seg_first, nslots) > tile_begin) --seg_first;
                int last = unit0;
                while (last + 1 < nslots && sk_range_begin(p, last + 1, nslots) < tile_end) ++last;
                seg_count = last - seg_first + 1;
            }
            bool waited_contrib = false, parked = false;
            unsigned int *ticket = nullptr;
            if (SK && t.shared && seg_count > 1 && row0 < q.M && t.tn * BN + chunk_lo * 32 < q.N) {
                const size_t region = (static_cast<size_t>(t.tile - p.sk_first_tile) * CG + cta_rank) * kEpiWarps + ew;
                ticket = p.sk_flags + static_cast<size_t>(gridDim.x) * 2 * kEpiWarps + region;
                unsigned int old = 0;
                if (lane == 0) old = atomicAdd(ticket, 1u);
                old = __shfl_sync(0xffffffffu, old, 0);
                reducer = old == static_cast<unsigned int>(seg_count - 1);
            }
            const bool park_it = SK && t.shared && seg_count > 1 && !reducer;
            // The reducer's list of the tile's other units, in slot order: index of their parking place
            // ((cta * 2 + place) * warps + warp, also the index of its ready flag).
            size_t others[kSkMaxShare - 1];
            int n_others = 0, n_before = 0;
            if (SK && reducer) {
                const long long tile_begin = static_cast<long long>(t.tile - p.sk_first_tile) * (q.fold * q.kiters);
                for (int j = seg_first; j < seg_first + seg_count; ++j) {
                    if (j == unit0) continue;
                    const int idx = (j == seg_first && sk_range_begin(p, j, nslots) < tile_begin) ? 1 : 0;
                    others[n_others++] = (static_cast<size_t>(j * CG + static_cast<int>(cta_rank)) * 2 + idx) * kEpiWarps + ew;
                    if (j < unit0) ++n_before;
                }
            }
            if constexpr (RUN) {
                __syncwarp();                          // tcgen05.ld is warp-collective
                const long long t_ld0 = p.prof ? clock64() : 0;
                if (!later_piece) {
#pragma unroll
                    for (int c = 0; c < CHUNKS; ++c) tmem_ld32_issue(tbase + (chunk_lo + c) * 32, run[c]);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int c = 0; c < 2 * CHUNKS; ++c) {
                        uint32_t x[16];
                        tmem_ld16_issue(tbase + chunk_lo * 32 + c * 16, x);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            uint32_t &r = run[c / 2][(c & 1) * 16 + e];
                            r = __float_as_uint(__uint_as_float(r) + __uint_as_float(x[e]));
                        }
                    }
                }
                // the accumulator has been read: the MMA warp may refill it while this sum goes out
                auto release = [&](int slot) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 2 && cta_rank != 0) mbar_arrive_cta(bar_acc_empty + 8u * slot, 0u);
                        else mbar_arrive(bar_acc_empty + 8u * slot);
                    }
                };
                release(buf);
                if constexpr (TWO) {
                    const float small_scale = wide ? 1.f : 1.f / (1 << kHalfLoShift);
#pragma unroll
                    for (int c = 0; c < CHUNKS; ++c) {
                        uint32_t x[32];
                        tmem_ld32_issue(tbase + BN + (chunk_lo + c) * 32, x);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e)
                            run[c][e] = __float_as_uint(fmaf(__uint_as_float(x[e]), small_scale, __uint_as_float(run[c][e])));
                    }
                    release(1);
                }
                if (p.prof) t_ld += clock64() - t_ld0;
                ++acc_it;
                if (!last_piece) continue;
            }
            if (row0 < q.M) {
#pragma unroll(RUN ? CHUNKS : 1)
                for (int c = 0; c < CHUNKS; ++c) {
                    const int chunk = chunk_lo + c;
                    const int col0 = t.tn * BN + chunk * 32;
                    if (col0 >= q.N) break;           // warp-uniform
                    uint32_t loaded[32];
                    uint32_t (&v)[32] = RUN ? run[RUN ? c : 0] : loaded;
                    if constexpr (!RUN) {
                        __syncwarp();                  // tcgen05.ld is warp-collective
                        const long long t_ld0 = p.prof ? clock64() : 0;
                        tmem_ld32_issue(tbase + chunk * 32, v);
                        tmem_ld_wait();
                        if (p.prof) t_ld += clock64() - t_ld0;
                    }
                    if constexpr (HALF) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * unscale);
                    }
                    if (park_it) {
                        // [j][lane] order: one instruction of the warp writes 512 contiguous bytes
                        float4 *dst = reinterpret_cast<float4 *>(
                            p.sk_partial + (((static_cast<size_t>(my_cta) * 2 + t.park) * kEpiWarps + ew) * CHUNKS + (chunk - chunk_lo)) * 1024) + lane;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            __stcg(dst + j * 32, make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                        __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
                        parked = true;
                        continue;
                    }
                    if (SK && reducer) {
                        if (!waited_contrib) {
                            // Bounded wait for the ready flag of every other unit of the tile (they took their
                            // tickets earlier, so they are at most one parking pass behind).
                            for (int o = 0; ok && o < n_others; ++o) {
                                const unsigned int *flag = p.sk_flags + others[o];
                                const long long tw0 = clock64();
                                unsigned int seen = 0;
                                while (true) {
                                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
                                    if (seen != 0u) break;
                                    if (*abort_flag || clock64() - tw0 > p.wait_cycles) {
                                        *abort_flag = 1u;
                                        atomicCAS(p.err, 0u, 0x600u);
                                        ok = false;
                                        break;
                                    }
                                }
                            }
                            ok = __all_sync(0xffffffffu, ok);
                            waited_contrib = true;
                            if (!ok) break;
                        }
                        // Sum in slot (= ascending k) order; this warp's own accumulator takes its place in it.
                        // Each parked tile is fetched with independent 16-byte loads, half a chunk at a time.
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float4 pre[4];
                            for (int o = 0; o < n_before; ++o) {
                                const float4 *src = reinterpret_cast<const float4 *>(
                                                        p.sk_partial + (others[o] * CHUNKS + (chunk - chunk_lo)) * 1024) + h * 128 + lane;
                                float4 x[4];
#pragma unroll
                                for (int u = 0; u < 4; ++u) x[u] = __ldcg(src + u * 32);
#pragma unroll
                                for (int u = 0; u < 4; ++u) {
                                    if (o == 0) pre[u] = x[u];
                                    else { pre[u].x += x[u].x; pre[u].y += x[u].y; pre[u].z += x[u].z; pre[u].w += x[u].w; }
                                }
                            }
                            if (n_before > 0) {
#pragma unroll
                                for (int u = 0; u < 4; ++u) {
                                    const int b = 16 * h + 4 * u;
                                    v[b + 0] = __float_as_uint(pre[u].x + __uint_as_float(v[b + 0]));
                                    v[b + 1] = __float_as_uint(pre[u].y + __uint_as_float(v[b + 1]));
                                    v[b + 2] = __float_as_uint(pre[u].z + __uint_as_float(v[b + 2]));
                                    v[b + 3] = __float_as_uint(pre[u].w + __uint_as_float(v[b + 3]));
                                }
                            }
                            for (int o = n_before; o < n_others; ++o) {
                                const float4 *src = reinterpret_cast<const float4 *>(
                                                        p.sk_partial + (others[o] * CHUNKS + (chunk - chunk_lo)) * 1024) + h * 128 + lane;
                                float4 x[4];
#pragma unroll
                                for (int u = 0; u < 4; ++u) x[u] = __ldcg(src + u * 32);
#pragma unroll
                                for (int u = 0; u < 4; ++u) {
                                    const int b = 16 * h + 4 * u;
                                    v[b + 0] = __float_as_uint(__uint_as_float(v[b + 0]) + x[u].x);
                                    v[b + 1] = __float_as_uint(__uint_as_float(v[b + 1]) + x[u].y);
                                    v[b + 2] = __float_as_uint(__uint_as_float(v[b + 2]) + x[u].z);
                                    v[b + 3] = __float_as_uint(__uint_as_float(v[b + 3]) + x[u].w);
                                }
                            }
                        }
                    }
                    // Stages the 32 values of this lane's row into the warp's next patch and hands the
                    // patch to the TMA unit (store, or reduce-add for C += ...).  `gelu`: applied to the staged row, four
                    // elements at a time: unrolled over the row's registers its code, which few calls run, took the place of the
                    // others' in the instruction cache (100 x [256 x 512 x 64] 19.3 -> 21.7 us).
                    auto emit = [&](const CUtensorMap *map, bool reduce, bool gelu = false) {
                        const long long t_wg0 = p.prof ? clock64() : 0;
                        if (lane == 0 && in_flight == p.epi_patches) {   // the patch must have been read by its store
                            if (p.epi_patches == 1) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                            else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                            --in_flight;
                        }
                        __syncwarp();
                        if (p.prof) t_wg += clock64() - t_wg0;
                        if (!RUN && p.transpose_out) {
                            // patch row j = this chunk's column j, float `lane` of it = this lane's row:
                            // the 32 lanes fill one 128-byte line per store, conflict-free
                            uint8_t *dst = my_stage + patch * kEpiBufBytes + ((lane & 3) << 2);
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                *reinterpret_cast<uint32_t *>(dst + j * 128 + (((lane >> 2) ^ (j & 7)) << 4)) = v[j];
                        } else {
                            uint8_t *dst = my_stage + patch * kEpiBufBytes + lane * 128;
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                *reinterpret_cast<float4 *>(dst + ((j ^ (lane & 7)) << 4)) =
                                    make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                            if (gelu) {
#pragma unroll 1
                                for (int j = 0; j < 8; ++j) {
                                    float4 *const at = reinterpret_cast<float4 *>(dst + ((j ^ (lane & 7)) << 4));   // no bank conflicts
                                    const float4 x = *at;
                                    *at = make_float4(gelu_tanh(x.x), gelu_tanh(x.y), gelu_tanh(x.z), gelu_tanh(x.w));
                                }
                            }
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            const uint32_t src = smem_u32(my_stage + patch * kEpiBufBytes);
                            const int c0 = part ? chunk * 32 : (!RUN && p.transpose_out) ? row0 : col0;
                            const int c1 = part ? static_cast<int>(cta_rank) * BM + quarter * 32 : (!RUN && p.transpose_out) ? col0 : row0;
                            const int c2 = part ? t.part : cbatch;
                            if (reduce) tma_reduce_add_5d(map, src, c0, c1, c2);
                            else tma_store_5d(map, src, c0, c1, c2);
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                            ++in_flight;
                        }
                        if (++patch == p.epi_patches) patch = 0;
                    };
                    const bool do_act = (!RUN || HALF) && fuse && q.act != 0;          // host guarantees use_tma in this mode
                    if (do_act && q.store_pre) emit(&w.C, false);    // the raw product, what the tape saves
                    if (fuse && q.bias != nullptr && add_piece) {
                        // the bias went in with the first piece
                    } else if (!RUN && fuse && q.bias != nullptr && p.transpose_out) {
                        const float b = row0 + lane < q.M ? __ldg(q.bias + row0 + lane) : 0.f;   // one bias value per row here
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + b);
                    } else if (fuse && q.bias != nullptr) {
                        if (bias_vec && col0 + 32 <= q.N) {
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float4 b = __ldg(reinterpret_cast<const float4 *>(q.bias + col0) + j);
                                v[4 * j + 0] = __float_as_uint(__uint_as_float(v[4 * j + 0]) + b.x);
                                v[4 * j + 1] = __float_as_uint(__uint_as_float(v[4 * j + 1]) + b.y);
                                v[4 * j + 2] = __float_as_uint(__uint_as_float(v[4 * j + 2]) + b.z);
                                v[4 * j + 3] = __float_as_uint(__uint_as_float(v[4 * j + 3]) + b.w);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (col0 + j < q.N) v[j] = __float_as_uint(__uint_as_float(v[j]) + __ldg(q.bias + col0 + j));
                        }
                    }
                    if (do_act) {
                        emit(&w.D, false, true);
                    } else if (part) {
                        emit(&w.P, add_piece);
                    } else if ((RUN && !HALF) || use_tma) {
                        emit(&w.C, (q.epi_mode == kEpiTmaReduce && fuse) || add_piece);
                    } else {
                        float *out0 = fuse ? q.C + static_cast<long long>(t.bt) * q.c_bstride + static_cast<long long>(row0) * q.ldc
                                           : q.partial + (static_cast<long long>(cbatch) * q.M + row0) * q.partial_ld;
                        const long long pitch = fuse ? q.ldc : q.partial_ld;
                        const bool add = (fuse && q.accumulate) || add_piece;
                        if (q.epi_mode == kEpiVectorStores && col0 + 32 <= q.N) {
                            // Each lane owns one row: four 32-byte stores write whole sectors, no staging.
                            if (row0 + lane >= q.M) continue;
                            float *dst = out0 + lane * pitch + col0;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float y[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e) y[e] = __uint_as_float(v[8 * j + e]);
                                if (add) {
                                    float o[8];
                                    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                                 : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]),
                                                   "=f"(o[6]), "=f"(o[7])
                                                 : "l"(dst + 8 * j));
#pragma unroll
                                    for (int e = 0; e < 8; ++e) y[e] += o[e];
                                }
                                asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + 8 * j),
                                             "f"(y[0]), "f"(y[1]), "f"(y[2]), "f"(y[3]), "f"(y[4]), "f"(y[5]), "f"(y[6]),
                                             "f"(y[7])
                                             : "memory");
                            }
                            continue;
                        }
                        // Rows that are not 16-byte aligned (an odd width): the patch is turned in the warp's staging
                        // buffer, so that every store covers 32 neighbouring columns of one row.  Stored straight from
                        // the accumulator's row-per-lane order each instruction touched 32 rows (attention scores of
                        // length 333: 75 us a product).
                        uint8_t *mine = my_stage + lane * 128;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            *reinterpret_cast<float4 *>(mine + ((j ^ (lane & 7)) << 4)) =
                                make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                            __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                        __syncwarp();
                        const int rows = min(32, q.M - row0);
                        if (col0 + lane < q.N) {
                            float *dst = out0 + col0 + lane;
                            const uint8_t *src = my_stage + ((lane & 3) << 2);
#pragma unroll 2
                            for (int r4 = 0; r4 < 32; r4 += 4) {
                                float y[4];
#pragma unroll
                                for (int r = 0; r < 4; ++r)
                                    y[r] = *reinterpret_cast<const float *>(src + (r4 + r) * 128 + (((lane >> 2) ^ ((r4 + r) & 7)) << 4));
                                if (add) {
#pragma unroll
                                    for (int r = 0; r < 4; ++r) y[r] += r4 + r < rows ? dst[(r4 + r) * pitch] : 0.f;
                                }
#pragma unroll
                                for (int r = 0; r < 4; ++r)
                                    if (r4 + r < rows) dst[(r4 + r) * pitch] = y[r];
                            }
                        }
                        __syncwarp();                  // the staging buffer is free again
                    }
                }
            }
            if (!ok) break;
            if (parked) {
                // publish: every lane's stores are fenced, then one release store of the ready flag
                __threadfence();
                __syncwarp();
                if (lane == 0) {
                    unsigned int *flag = p.sk_flags + ((static_cast<size_t>(my_cta) * 2 + t.park) * kEpiWarps + ew);
                    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(1u) : "memory");
                }
            } else if (SK && reducer) {
                // every lane has read the parked tiles: ticket and ready flags go back to zero for the next launch
                __syncwarp();
                if (lane == 0) {
                    *ticket = 0u;
                    if (waited_contrib)
                        for (int o = 0; o < n_others; ++o) p.sk_flags[others[o]] = 0u;
                }
            }
            if constexpr (!RUN) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2 && cta_rank != 0) mbar_arrive_cta(bar_acc_empty + 8u * buf, 0u);
                    else mbar_arrive(bar_acc_empty + 8u * buf);
                }
                ++acc_it;
            }
        }
        }
        // The staging patches must have been read before the CTA gives up its shared memory; the global
        // writes themselves complete with the grid like any other store.
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        if (p.prof && warp == EPI0 && lane == 0) {
            atomicAdd(p.prof + 4, static_cast<unsigned long long>(waited));
            atomicAdd(p.prof + 7, static_cast<unsigned long long>(t_wg));
            atomicAdd(p.prof + 1, static_cast<unsigned long long>(t_ld));
        }
    } else {
    if constexpr (RUN) {
        if (TWO) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTwoIssue));
        else if (warp < SPLIT0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RegShare<MODE>::kIssue));
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RegShare<MODE>::kSplit));
    }
    if (warp == 0 || (HALF && warp == SPLIT0 + 1)) {
        // ------------------------------------------------------------ TMA producer
        // The whole warp runs the loop; one elected lane issues the copies.  HALF: a stage holds a third of the time it holds
        // in 3xTF32, so a second warp issues B's copies (the first arms the barrier).
        const bool loads_a = !HALF || warp == 0, loads_b = !HALF || warp != 0;
        {
            int stage = 0;
            uint32_t phase = 0;
            int armed = 0;
            bool ok = true;
            long long waited = 0;
            constexpr uint32_t CHUNK_BYTES = 128u * BK;   // one 32-wide MN chunk: BK k-rows of 128 bytes
            const uint32_t dstA0 = smem_u32(stage_base);
            uint32_t dstA = dstA0;
#pragma unroll                             // parameters at constant addresses, so that what an MMA or a copy takes stays uniform
            for (int prod = 0; prod < product_slots(MODE); ++prod) {
            if (!ok || prod >= products) break;
            const Product &w = g.s[HALF ? prod : 0];
            const KParams &q = HALF ? w.p : p;
            const int a_mode = q.a_mode, b_mode = q.b_mode, kiters = q.kiters;
            WorkIter wi = work_begin(q, first_unit(prod), unit_step);
            TileCoord t;
            while (ok && work_next<TAIL>(q, wi, t)) {
                int f = 0, kk = t.it0;
                if (t.it0 >= q.kiters) {
                    f = t.it0 / q.kiters;
                    kk = t.it0 - f * q.kiters;
                }
                int a0, a1, a2, b0, b1, b2;
                batch_coords(t.bt * q.fold + f, q.a_batch, q.a_d1, q.a_d2, q.fd_a_cnt, q.fd_a_d1, q.fd_a_d2, a0, a1, a2);
                batch_coords(t.bt * q.fold + f, q.b_batch, q.b_d1, q.b_d2, q.fd_b_cnt, q.fd_b_d1, q.fd_b_d2, b0, b1, b2);
                const int rowA = t.tm * (BM * CG) + static_cast<int>(cta_rank) * BM;
                const int rowB = t.tn * BN + static_cast<int>(cta_rank) * BNL;
                if constexpr (HALF) {
                    // The planes of a k-block are staged one after the other, each in a stage of its own.  The plane is the map's
                    // second batch coordinate.
                    for (int it = t.it0; ok && it < t.it1; ++it) {
                        for (int plane = 0; plane < planes; ++plane) {
                            ok = mbar_wait_warp(bar_empty + 8u * stage, phase ^ 1u, abort_flag, p.err, 0x100u | stage, waited, timed, p.wait_cycles);
                            if (!ok) break;
                            const uint32_t full = bar_full + 8u * stage;
                            ++armed;
                            if (elect_one()) {
                                if (loads_a) mbar_arrive_expect_tx(full, RAW_BYTES);
                                if (armed != p.withhold_at) {
                                    if (loads_a) load_half(a_mode, dstA, &w.A, full, kk * BK, rowA, a2, plane);
                                    if (loads_b) load_half(b_mode, dstA + A_BYTES, &w.B, full, kk * BK, rowB, b2, plane);
                                }
                            }
                            if (++stage == p.stages) { stage = 0; phase ^= 1u; dstA = dstA0; } else { dstA += STAGE_BYTES; }
                        }
                        if (++kk == kiters) {
                            kk = 0;
                            ++f;
                            if (q.fold > 1) {
                                batch_coords(t.bt * q.fold + f, q.a_batch, q.a_d1, q.a_d2, q.fd_a_cnt, q.fd_a_d1, q.fd_a_d2, a0, a1, a2);
                                batch_coords(t.bt * q.fold + f, q.b_batch, q.b_d1, q.b_d2, q.fd_b_cnt, q.fd_b_d1, q.fd_b_d2, b0, b1, b2);
                            }
                        }
                    }
                } else
                for (int it = t.it0; it < t.it1; ++it) {
                    ok = mbar_wait_warp(bar_empty + 8u * stage, phase ^ 1u, abort_flag, p.err, 0x100u | stage, waited, timed, p.wait_cycles);
                    if (!ok) break;
                    const uint32_t full = bar_full + 8u * stage;
                    const int k0 = kk * BK;
                    ++armed;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(full, A_BYTES + static_cast<uint32_t>(q.b_rows_live) * BK * 4u);
                        if (armed != p.withhold_at) {        // test hook: a stage that is armed and never filled
                            load_operand(q.a_mode, dstA, &w.A, full, k0, rowA, BM / 32, CHUNK_BYTES, a0, a1, a2);
                            load_operand(q.b_mode, dstA + A_BYTES, &w.B, full, k0, rowB, BNL / 32, CHUNK_BYTES, b0, b1, b2);
                        }
                    }
                    if (++stage == p.stages) { stage = 0; phase ^= 1u; dstA = dstA0; } else { dstA += STAGE_BYTES; }
                    if (++kk == q.kiters) {
                        kk = 0;
                        ++f;
                        if (q.fold > 1) {
                            batch_coords(t.bt * q.fold + f, q.a_batch, q.a_d1, q.a_d2, q.fd_a_cnt, q.fd_a_d1, q.fd_a_d2, a0, a1, a2);
                            batch_coords(t.bt * q.fold + f, q.b_batch, q.b_d1, q.b_d2, q.fd_b_cnt, q.fd_b_d1, q.fd_b_d2, b0, b1, b2);
                        }
                    }
                }
            }
            }
            if (!ok) {
                // Aborting: let the copies already issued land before the CTA exits.
                const int pending = min(armed, p.stages);
                for (int i = 0; i < pending; ++i) {
                    if (--stage < 0) { stage = p.stages - 1; phase ^= 1u; }
                    const long long t0 = clock64();
                    while (!mbar_try_wait(bar_full + 8u * stage, phase) && clock64() - t0 < p.wait_cycles / 8) {}
                }
            }
            if (p.prof && lane == 0 && loads_a) atomicAdd(p.prof + 0, static_cast<unsigned long long>(waited));
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // The whole warp runs the loop; one elected lane issues each MMA and commit.  In a CTA pair
        // only the leader's warp issues (its MMAs drive both SMs); the peer's warp just holds TMEM.
        if (CG == 1 || cta_rank == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int acc_it = 0;
            bool ok = true;
            long long waited = 0, waited_acc = 0;
            bool next_ready = false;                   // the stage about to be consumed was already seen complete
            const uint32_t sa0 = smem_u32(stage_base);
#pragma unroll                             // parameters at constant addresses, so that what an MMA or a copy takes stays uniform
            for (int prod = 0; prod < product_slots(MODE); ++prod) {
            if (!ok || prod >= products) break;
            const KParams &q = HALF ? g.s[prod].p : p;
            const uint32_t a_lo0 = ((sa0 >> 4) & 0x3FFFu) | q.a_desc_lbo;
            const uint32_t b_lo0 = (((sa0 + A_BYTES) >> 4) & 0x3FFFu) | q.b_desc_lbo;
            uint32_t a_lo = a_lo0 + static_cast<uint32_t>(stage) * STAGE16, b_lo = b_lo0 + static_cast<uint32_t>(stage) * STAGE16;
            const uint32_t a_hi = q.a_desc_hi, b_hi = q.b_desc_hi;
            const uint32_t a_ks = q.a_kstep, b_ks = q.b_kstep;
            const uint32_t idesc = HALF && wide ? q.idesc | (1u << 7) | (1u << 10) : q.idesc;     // bf16 operands
            // A lone CTA in single-pass mode consumes the TMA barrier directly; otherwise the split warps
            // (of both CTAs, for a pair) announce the stage on the leader's barrier.
            const uint32_t ready0 = (FAST && CG == 1) ? bar_full : bar_xform;
            WorkIter wi = work_begin(q, first_unit(prod), unit_step);
            TileCoord wt;
            while (ok && work_next<TAIL>(q, wi, wt)) {
                const int iters = wt.it1 - wt.it0;
                const int buf = TWO ? 0 : acc_it & 1;
                const uint32_t acc_phase = TWO ? acc_it & 1 : (acc_it >> 1) & 1;
                ok = mbar_wait_warp(bar_acc_empty + 8u * buf, acc_phase ^ 1u, abort_flag, p.err, 0x200u | buf, waited_acc, timed, p.wait_cycles);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * BN);
                uint32_t accumulate = 0;
                if constexpr (HALF) {
                    auto next = [&] {
                        if (++stage == p.stages) { stage = 0; phase ^= 1u; a_lo = a_lo0; b_lo = b_lo0; }
                        else { a_lo += STAGE16; b_lo += STAGE16; }
                    };
                    // Compiled for each number of planes: as a run-time number it cost a tenth of the pipe (8192^3: 27.1 cycles per
                    // element of a tile instead of 24.4).
                    auto k_loop = [&](auto plane_count) {
                    constexpr int PLANES = decltype(plane_count)::value;
                    constexpr bool WIDE = PLANES > (TWO ? 2 : 1);
                    for (int it = 0; it < iters; ++it) {
                        ok = mbar_wait_warp(ready0 + 8u * stage, phase, abort_flag, p.err, 0x300u | stage, waited, timed, p.wait_cycles);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t hi_stage = static_cast<uint32_t>(stage), ah = a_lo, bh = b_lo;
                        if (elect_one()) {
#pragma unroll
                            for (int ks = 0; ks < KSTEPS; ++ks)
                                umma_f16_pair(d_tmem, ah + ks * a_ks, a_hi, bh + ks * b_ks, b_hi, idesc, ks == 0 ? accumulate : 1u);
                            if (PLANES == 1) umma_commit_pair(bar_empty + 8u * hi_stage);
                        }
                        __syncwarp();
                        next();
                        // The products with the planes below hi: into an accumulator of their own (TWO) or the same.
                        uint32_t small_acc = TWO ? accumulate : 1u;
#pragma unroll
                        for (int plane = 1; plane < PLANES; ++plane) {
                            ok = mbar_wait_warp(ready0 + 8u * stage, phase, abort_flag, p.err, 0x300u | stage, waited, timed, p.wait_cycles);
                            if (!ok) break;
                            if (TWO && it == 0 && plane == 1) {     // its accumulator comes free a little later than the other
                                ok = mbar_wait_warp(bar_acc_empty + 8u, acc_phase ^ 1u, abort_flag, p.err, 0x201u, waited_acc, timed, p.wait_cycles);
                                if (!ok) break;
                            }
                            tc_fence_after();
                            const uint32_t d_small = d_tmem + (TWO ? BN : 0);
                            if (elect_one()) {
#pragma unroll
                                for (int ks = 0; ks < KSTEPS; ++ks) {
                                    umma_f16_pair(d_small, a_lo + ks * a_ks, a_hi, bh + ks * b_ks, b_hi, idesc, ks == 0 ? small_acc : 1u);
                                    umma_f16_pair(d_small, ah + ks * a_ks, a_hi, b_lo + ks * b_ks, b_hi, idesc, 1u);
                                    if (TWO && WIDE && plane == 1)
                                        umma_f16_pair(d_small, a_lo + ks * a_ks, a_hi, b_lo + ks * b_ks, b_hi, idesc, 1u);
                                }
                                umma_commit_pair(bar_empty + 8u * stage);
                                if (plane + 1 == PLANES) umma_commit_pair(bar_empty + 8u * hi_stage);
                            }
                            __syncwarp();
                            small_acc = 1u;
                            next();
                        }
                        if (!ok) break;
                        accumulate = 1u;
                    }
                    };
                    if (wide) k_loop(std::integral_constant<int, TWO ? 3 : 2>{});
                    else k_loop(std::integral_constant<int, TWO ? 2 : 1>{});
                    if (ok && elect_one()) umma_commit_pair(bar_acc_full + 8u * buf);
                    __syncwarp();
                    if (!ok) break;
                    ++acc_it;
                } else
                {
                for (int it = 0; it < iters; ++it) {
                    if (!next_ready) {
                        ok = mbar_wait_warp(ready0 + 8u * stage, phase, abort_flag, p.err, 0x300u | stage, waited, timed, p.wait_cycles);
                        if (!ok) break;
                    }
                    tc_fence_after();
                    // Look at the following stage now; the answer is used after this stage's MMAs are
                    // queued, so the barrier read overlaps them (narrow tiles retire an MMA every 32
                    // cycles and would otherwise drain the queue during the wait).
                    const int nstage = stage + 1 == p.stages ? 0 : stage + 1;
                    const uint32_t peek = mbar_test_wait(ready0 + 8u * nstage, stage + 1 == p.stages ? phase ^ 1u : phase);
                    // This warp's own instruction count sets the pace of narrow tiles (an MMA retires every
                    // 32 cycles there): one election guards the whole k-block's MMAs and its stage commit
                    // (one election per MMA measured 12 % slower on the attention-shaped products; wide
                    // tiles measured the same either way).
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < KSTEPS; ++ks) {
                            const uint32_t ak = a_lo + ks * a_ks, bk = b_lo + ks * b_ks;
                            const uint32_t acc_first = ks == 0 ? accumulate : 1u;
                            if constexpr (TA) {
                                const uint32_t at = tmem_base + TA_COL0 + static_cast<uint32_t>(stage) * TA_SLOT + ks * 8;
                                umma_tf32_ts(d_tmem, at + BK, bk, b_hi, idesc, acc_first);
                                umma_tf32_ts(d_tmem, at, bk + LO16, b_hi, idesc, 1u);
                                umma_tf32_ts(d_tmem, at, bk, b_hi, idesc, 1u);
                            } else if constexpr (HALF) {
                            } else if constexpr (CG == 2 && FAST) {
                                umma_tf32_pair(d_tmem, ak, a_hi, bk, b_hi, idesc, acc_first);
                            } else if constexpr (CG == 2) {
                                umma_tf32_pair(d_tmem, ak + LO16, a_hi, bk, b_hi, idesc, acc_first);
                                umma_tf32_pair(d_tmem, ak, a_hi, bk + LO16, b_hi, idesc, 1u);
                                umma_tf32_pair(d_tmem, ak, a_hi, bk, b_hi, idesc, 1u);
                            } else if constexpr (FAST) {
                                umma_tf32(d_tmem, ak, a_hi, bk, b_hi, idesc, acc_first);
                            } else {
                                umma_tf32(d_tmem, ak + LO16, a_hi, bk, b_hi, idesc, acc_first);
                                umma_tf32(d_tmem, ak, a_hi, bk + LO16, b_hi, idesc, 1u);
                                umma_tf32(d_tmem, ak, a_hi, bk, b_hi, idesc, 1u);
                            }
                        }
                        if constexpr (CG == 2) umma_commit_pair(bar_empty + 8u * stage);
                        else umma_commit(bar_empty + 8u * stage);
                    }
                    accumulate = 1u;
                    next_ready = __all_sync(0xffffffffu, peek != 0u);
                    if (++stage == p.stages) {
                        stage = 0; phase ^= 1u; a_lo = a_lo0; b_lo = b_lo0;
                    } else {
                        a_lo += STAGE16; b_lo += STAGE16;
                    }
                }
                if (!ok) break;
                if constexpr (CG == 2) { if (elect_one()) umma_commit_pair(bar_acc_full + 8u * buf); }
                else { if (elect_one()) umma_commit(bar_acc_full + 8u * buf); }
                ++acc_it;
                }
            }
            }
            if (p.prof && lane == 0) {
                atomicAdd(p.prof + 1, static_cast<unsigned long long>(waited_acc));
                atomicAdd(p.prof + 2, static_cast<unsigned long long>(waited));
            }
        }
    } else if (RUN && !TWO && warp < SPLIT0) {
        // idle: the rest of the first warpgroup
    } else {
        // ------------------------------------------------------------ hi/lo split
        // In single-pass mode there is nothing to split; for a CTA pair these warps still relay "my
        // CTA's tile has landed" to the leader's barrier.
        if (!FAST || CG == 2) {
            // With A in tensor memory one k-block is a serial chain per warp (barrier wake-up, loads, split, tensor-
            // memory stores and their completion, fence, arrival: ~600 cycles, measured) that the eight warps walk in
            // lockstep, each on one k-half of its lane quarter's rows (SG = 1).  With SG = 2 they work as two groups
            // of four (one warp per lane quarter) on alternate k-blocks instead: twice the work per warp and k-block,
            // two k-blocks in flight.  The host picks SG = 2 for long contractions.
            static_assert(SG == 1 || (SG == 2 && TA), "two split groups exist for the tensor-memory A variants only");
            constexpr int GROUPS = SG;
            const int group = TA ? (warp - SPLIT0) >> 2 : 0;   // SG = 1: the k-half this warp splits; SG = 2: its group
            const int tid = (threadIdx.x - 32 * SPLIT0) & (32 * NS / GROUPS - 1);   // index within the group
            int stage = 0;
            int kb = 0;                                   // k-blocks this CTA has seen: the group takes those of its parity
            uint32_t phase = 0;
            bool ok = true;
            long long waited = 0;
            constexpr int N4 = (TA ? B_BYTES : RAW_BYTES) >> 4;   // float4 count of what gets a lo copy
            constexpr int NT = 32 * NS / GROUPS;          // split threads that share one k-block
            constexpr int PER = (N4 + NT - 1) / NT;       // float4s per thread (the last round may be partial)
            constexpr bool EXACT = N4 % NT == 0;
            constexpr int U = !EXACT ? 1 : (PER % 4 == 0) ? 4 : (PER % 2 == 0 ? 2 : 1);
            if (HALF && warp != SPLIT0) ok = false;           // one warp relays there
#pragma unroll                             // parameters at constant addresses, so that what an MMA or a copy takes stays uniform
            for (int prod = 0; prod < product_slots(MODE); ++prod) {
            if (!ok || prod >= products) break;
            const KParams &q = HALF ? g.s[prod].p : p;
            WorkIter wi = work_begin(q, first_unit(prod), unit_step);
            TileCoord wt;
            while (ok && work_next<TAIL>(q, wi, wt)) {
                int iters = wt.it1 - wt.it0;
                if (HALF) iters *= planes;                        // each takes a stage
                for (int it = 0; it < iters; ++it) {
                    if (SG == 2 && ((kb++ & 1) != group)) {    // the other group's k-block
                        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
                        continue;
                    }
                    ok = mbar_wait(bar_full + 8u * stage, phase, abort_flag, p.err, 0x400u | stage, waited, timed, p.wait_cycles);
                    if (!ok) break;
                    if constexpr (TA) {
                      // A: this thread owns a row (lane quarter of its warp), 16 of the 32 k columns at a time.
                      const uint8_t *sa = stage_base + static_cast<size_t>(stage) * STAGE_BYTES;
                      const int row = (warp & 3) * 32 + lane;
#pragma unroll
                      for (int h = 0; h < SG; ++h) {
                        const int half = SG == 2 ? h : group;
                        uint32_t hi[16], lo16[16];
                        if (q.a_mode == kKMajor) {
                            // 128-byte rows, 16-byte chunk c of row r sits at chunk c ^ (r % 8)
                            const uint8_t *rp = sa + row * 128;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float4 x = *reinterpret_cast<const float4 *>(rp + (((half * 4 + j) ^ (row & 7)) << 4));
                                hi[4 * j + 0] = __float_as_uint(x.x); hi[4 * j + 1] = __float_as_uint(x.y);
                                hi[4 * j + 2] = __float_as_uint(x.z); hi[4 * j + 3] = __float_as_uint(x.w);
                            }
                        } else {
                            // 32-row chunks of BK k-lines of 128 bytes; 32-byte atom a of k-line k sits at a ^ (k % 4)
                            const uint8_t *cp = sa + (row >> 5) * (128 * BK) + ((row & 7) << 2);
                            const int atom = (row & 31) >> 3;
#pragma unroll
                            for (int kk = 0; kk < 16; ++kk) {
                                const int k = half * 16 + kk;
                                hi[kk] = *reinterpret_cast<const uint32_t *>(cp + k * 128 + ((atom ^ (k & 3)) << 5));
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            const float x = __uint_as_float(hi[e]);
                            hi[e] &= 0xFFFFE000u;
                            lo16[e] = __float_as_uint(x - __uint_as_float(hi[e]));
                        }
                        const uint32_t ta = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + TA_COL0 +
                                            static_cast<uint32_t>(stage) * TA_SLOT + half * 16;
                        __syncwarp();                      // tcgen05.st is warp-collective
                        tmem_st16(ta, hi);
                        tmem_st16(ta + BK, lo16);
                      }
                    }
                    // TA: only the B tile gets a lo copy in shared memory (it sits right behind the raw B tile).
                    const float4 *raw = reinterpret_cast<const float4 *>(stage_base + static_cast<size_t>(stage) * STAGE_BYTES +
                                                                         (TA ? A_BYTES : 0));
                    float4 *lo = const_cast<float4 *>(raw) + N4;
                    // float4s that hold data: all of them, or A and the live rows of B
                    const int live4 = N4 - ((BNL - q.b_rows_live) * BK * 4 >> 4);
#pragma unroll
                    for (int g = 0; g < (FAST ? 0 : PER); g += U) {
                        float4 v[U];
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (tid + (g + u) * NT < live4) v[u] = raw[tid + (g + u) * NT];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            if (tid + (g + u) * NT >= live4) continue;
                            float4 l;
                            l.x = v[u].x - __uint_as_float(__float_as_uint(v[u].x) & 0xFFFFE000u);
                            l.y = v[u].y - __uint_as_float(__float_as_uint(v[u].y) & 0xFFFFE000u);
                            l.z = v[u].z - __uint_as_float(__float_as_uint(v[u].z) & 0xFFFFE000u);
                            l.w = v[u].w - __uint_as_float(__float_as_uint(v[u].w) & 0xFFFFE000u);
                            lo[tid + (g + u) * NT] = l;
                        }
                    }
                    if constexpr (TA) {                       // the stores above complete while the B tile was split
                        tmem_st_wait();
                        tc_fence_before();
                    }
                    // Every thread publishes its writes to the async proxy; one lane per warp then arrives
                    // (a remote arrival crosses SMs, so they are kept to one per warp).
                    if (!FAST) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 2 && cta_rank != 0) mbar_arrive_cta(bar_xform + 8u * stage, 0u);
                        else mbar_arrive(bar_xform + 8u * stage);
                    }
                    if (++stage == p.stages) { stage = 0; phase ^= 1u; }
                }
            }
            }
            if (p.prof && tid == 0) atomicAdd(p.prof + 3, static_cast<unsigned long long>(waited));
        }
    }
    }

    tc_fence_before();
    __syncthreads();
    if (p.prof && threadIdx.x == 0) {
        atomicAdd(p.prof + 5, static_cast<unsigned long long>(clock64() - t_kernel0));
        atomicAdd(p.prof + 6, 1ull);
    }
    if constexpr (CG == 2) cluster_sync_all();   // both CTAs are done with the pair's TMEM and barriers
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        if constexpr (CG == 2)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                         : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                         : "memory");
    }
    // Stream order for whatever follows: this grid may not complete before the grid it ran beside has.
    if (p.dep_mode == 2 && threadIdx.x == 0) grid_dependency_wait();
}

// Divisors of the finish kernel: multiply-high and shift below 2^31 items, plain 64-bit beyond.
__device__ __forceinline__ uint32_t divisor(const FastDiv &f) { return f.d; }
__device__ __forceinline__ long long divisor(long long d) { return d; }
__device__ __forceinline__ unsigned divide(unsigned n, const FastDiv &f) { return static_cast<unsigned>(fd_div(static_cast<int>(n), f)); }
__device__ __forceinline__ long long divide(long long n, long long d) { return n / d; }
// Deterministic split-K finish: C = sum_s partial[s] (+ bias) (+ C), splits added in ascending order.
// One thread per 16-byte vector of the partials (rows of `pld` floats); the partials of four splits are in flight at a
// time.  VEC: the output's rows are whole aligned vectors too.  Otherwise (an odd width) a warp turns its 128
// columns through shared memory, so that its stores cover 32 neighbouring elements.
// dep_mode 1 / 2: first / second of two finishes launched back to back that need nothing from each other; the second starts
// once every block of the first has seen the products complete, and waits for the first only before it ends (as the pair of
// products does; a backward of 1000 x 333 x 777: 5 us less than one after the other).
template <bool VEC, typename I, typename D>
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float *__restrict__ partial, float *__restrict__ C, long long ldc, long long c_bstride,
                     const float *__restrict__ bias, int accumulate, int splits, long long rows, D rows_per_batch, D vectors,
                     int M, int N, int dep_mode) {
    __shared__ float turn[VEC ? 1 : 256 * 4];
    if (dep_mode != 1) grid_dependency_trigger();
    if (dep_mode != 2) grid_dependency_wait();   // the partials come from the grids before this one
    if (dep_mode == 1) grid_dependency_trigger();
    const I per_row = static_cast<I>(divisor(vectors));
    const I items = static_cast<I>(rows) * per_row;
    const I item = static_cast<I>(blockIdx.x) * 256 + threadIdx.x;
    const long long slab = rows * per_row;       // in vectors
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (item < items) {
        const float4 *src = reinterpret_cast<const float4 *>(partial) + item;
        int sp = 0;
        for (; sp + 4 <= splits; sp += 4) {
            float4 t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) t[u] = __ldcg(src + (sp + u) * slab);
#pragma unroll
            for (int u = 0; u < 4; ++u) { acc.x += t[u].x; acc.y += t[u].y; acc.z += t[u].z; acc.w += t[u].w; }
        }
        for (; sp < splits; ++sp) {
            const float4 t = __ldcg(src + sp * slab);
            acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
        }
    }
    if (VEC) {
        if (item < items) {
            const I row = divide(item, vectors);
            const int col = static_cast<int>(item - row * per_row) * 4;
            const I bt = divide(row, rows_per_batch);
            const int m = static_cast<int>(row - bt * static_cast<I>(M));
            if (bias) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(bias + col));
                acc.x += b.x; acc.y += b.y; acc.z += b.z; acc.w += b.w;
            }
            float4 *out = reinterpret_cast<float4 *>(C + static_cast<long long>(bt) * c_bstride + static_cast<long long>(m) * ldc + col);
            if (accumulate) {
                const float4 c0 = *out;
                acc.x += c0.x; acc.y += c0.y; acc.z += c0.z; acc.w += c0.w;
            }
            *out = acc;
        }
    } else {
        const int lane = threadIdx.x & 31;
        float *mine = turn + (threadIdx.x & ~31) * 4;
        reinterpret_cast<float4 *>(mine)[lane] = acc;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = j * 32 + lane;                           // element within the warp's 128
            const I at = (item - lane) + e / 4;                    // its vector
            if (at >= items) continue;
            const I row = divide(at, vectors);
            const int col = static_cast<int>(at - row * per_row) * 4 + (e & 3);
            if (col >= N) continue;
            const I bt = divide(row, rows_per_batch);
            const int m = static_cast<int>(row - bt * static_cast<I>(M));
            float *out = C + static_cast<long long>(bt) * c_bstride + static_cast<long long>(m) * ldc + col;
            float y = mine[e];
            if (bias) y += __ldg(bias + col);
            if (accumulate) y += *out;
            *out = y;
        }
    }
    if (dep_mode == 2) grid_dependency_wait();
}

// Finish of a split tail: adds the `tail_ways` partial tiles of each of the last wave's tiles in ascending order and runs
// what the GEMM epilogue does to a whole tile (bias, C += ..., gelu into the second output).  grid = (tile rows / 4, tail
// tiles); a row of the tile is 64 vectors, two warps.
template <bool VEC>
__global__ void __launch_bounds__(256)
tail_finish_kernel(const float *__restrict__ partial, float *__restrict__ D, int bn, int tile_rows, int dep_mode,
                   const __grid_constant__ KParams p) {
    __shared__ float turn[VEC ? 1 : 256 * 4];
    if (dep_mode != 1) grid_dependency_trigger();
    const TileCoord t = decode_unit<kCutTiles>(p, p.tail_unit + static_cast<int>(blockIdx.y) * p.tail_ways);
    const int r = static_cast<int>(blockIdx.x) * 4 + (threadIdx.x >> 6), c4 = threadIdx.x & 63;
    const int row = t.tm * tile_rows + r, col = t.tn * bn + c4 * 4;
    if (dep_mode != 2) grid_dependency_wait();   // the partials come from the grids before this one
    if (dep_mode == 1) grid_dependency_trigger();
    struct AtEnd {                               // dep_mode 2: see splitk_reduce_kernel
        bool wait;
        __device__ ~AtEnd() { if (wait) grid_dependency_wait(); }
    } at_end{dep_mode == 2};
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < p.M && col < p.N) {
        const float4 *src = reinterpret_cast<const float4 *>(partial) +
                            ((static_cast<long long>(blockIdx.y) * p.tail_ways) * tile_rows + r) * (bn / 4) + c4;
        float4 x[4];
        const long long step = static_cast<long long>(tile_rows) * (bn / 4);
        for (int w0 = 0; w0 < p.tail_ways; w0 += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (w0 + u < p.tail_ways) x[u] = __ldcg(src + (w0 + u) * step);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (w0 + u < p.tail_ways) { acc.x += x[u].x; acc.y += x[u].y; acc.z += x[u].z; acc.w += x[u].w; }
        }
    }
    const long long at = static_cast<long long>(t.bt) * p.c_bstride + static_cast<long long>(row) * p.ldc;
    if (VEC) {
        if (row >= p.M || col >= p.N) return;
        float v[4] = {acc.x, acc.y, acc.z, acc.w};
        if (D && p.C) *reinterpret_cast<float4 *>(p.C + at + col) = acc;       // the raw product, what the tape saves
        if (p.bias) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] += __ldg(p.bias + col + e);
        }
        float4 *out = reinterpret_cast<float4 *>((D ? D : p.C) + at + col);
        if (D) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = gelu_tanh(v[e]);
        } else if (p.accumulate) {
            const float4 c0 = *out;
            v[0] += c0.x; v[1] += c0.y; v[2] += c0.z; v[3] += c0.w;
        }
        *out = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
    // rows that are not whole aligned vectors: a warp turns its 128 columns, so that a store covers 32 neighbours
    const int lane = threadIdx.x & 31;
    float *mine = turn + (threadIdx.x & ~31) * 4;
    reinterpret_cast<float4 *>(mine)[lane] = acc;
    __syncwarp();
    if (row >= p.M) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int cc = t.tn * bn + (threadIdx.x & 32) * 4 + j * 32 + lane;
        if (cc >= p.N) continue;
        float y = mine[j * 32 + lane];
        if (D && p.C) p.C[at + cc] = y;
        if (p.bias) y += __ldg(p.bias + cc);
        float *out = (D ? D : p.C) + at + cc;
        if (D) y = gelu_tanh(y);
        else if (p.accumulate) y += *out;
        *out = y;
    }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

// Encoded tensor maps are a pure function of (pointer, extents, strides, box, swizzle): a training loop calls with
// the same handful of buffers every step, so each host thread keeps the maps it has built (bounded; dropped
// wholesale when full) and an eager call pays a hash lookup instead of three or four driver encodes.
struct MapKey {
    const void *ptr;
    cuuint64_t dims[5];
    cuuint64_t strides[4];
    cuuint32_t box[5];
    int swz;                       // and the element type
    bool operator==(const MapKey &o) const { return memcmp(this, &o, sizeof(MapKey)) == 0; }
};
struct MapKeyHash {
    size_t operator()(const MapKey &k) const {
        static_assert(sizeof(MapKey) % 8 == 0, "hashed in 8-byte words");
        uint64_t h = 1469598103934665603ull;
        for (size_t i = 0; i < sizeof(MapKey); i += 8) {
            uint64_t w;
            memcpy(&w, reinterpret_cast<const unsigned char *>(&k) + i, 8);
            h = (h ^ w) * 0x9e3779b97f4a7c15ull;
            h ^= h >> 29;
        }
        return static_cast<size_t>(h);
    }
};
constexpr size_t kMapCacheEntries = 512;

CUresult encode(CUtensorMap *map, const void *ptr, const cuuint64_t *dims, const cuuint64_t *strides,
                const cuuint32_t *box, CUtensorMapSwizzle swz, CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_FLOAT32) {
    static thread_local std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
    static const bool use_cache = env_int("MNI_B200_MAP_CACHE", 1) != 0;
    MapKey key;
    memset(&key, 0, sizeof(key));                       // padding bytes take part in the comparison
    key.ptr = ptr;
    for (int i = 0; i < 5; ++i) { key.dims[i] = dims[i]; key.box[i] = box[i]; }
    for (int i = 0; i < 4; ++i) key.strides[i] = strides[i];
    key.swz = static_cast<int>(swz) + 256 * static_cast<int>(type);
    if (use_cache) {
        auto it = cache.find(key);
        if (it != cache.end()) { *map = it->second; return CUDA_SUCCESS; }
    }
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode_fn()(map, type, 5, const_cast<void *>(ptr), dims, strides, box,
                                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS && use_cache) {
        if (cache.size() >= kMapCacheEntries) cache.clear();
        cache.emplace(key, *map);
    }
    return r;
}

// Builds the tensor map of one operand and reports the OperandMode the kernel must use for it.
int make_operand_map(CUtensorMap *map, const Operand &op, int box_rows, int bk, int *mode) {
    if (!encode_fn()) return fail(MNI_B200_ERR_CUDA, "cuTensorMapEncodeTiled entry point not found");
    cuuint64_t dims[5];
    cuuint64_t strides[4];   // bytes, dims 1..4
    cuuint32_t box[5] = {1, 1, 1, 1, 1};
    // A size-1 dim never advances, but its stride must still be a positive multiple of 16 bytes.
    uint64_t span = 16;
    auto stride_or = [&](int64_t extent, int64_t stride_elems) -> cuuint64_t {
        return static_cast<cuuint64_t>((extent > 1 && stride_elems > 0) ? static_cast<uint64_t>(stride_elems) * 4u : span);
    };
    // 32-bit elements read MN-major by the tensor core use the 128-byte swizzle whose unit is a
    // 32-byte chunk, not the usual 16-byte chunk.
    const CUtensorMapSwizzle mn_swz = CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B;
    if (!op.k_major && op.rows % 32 == 0 && op.bshape[0] == 1 && env_int("MNI_B200_NO_SINGLE_BOX", 0) == 0) {
        // One box per tile: the MN dim is split into (32 contiguous floats, rows/32 chunks), giving the
        // smem order [chunk][k][32 floats] the MMA descriptor expects.
        dims[0] = 32;
        dims[1] = static_cast<cuuint64_t>(op.kdim);
        dims[2] = static_cast<cuuint64_t>(op.rows / 32);
        dims[3] = static_cast<cuuint64_t>(op.bshape[2]);
        dims[4] = static_cast<cuuint64_t>(op.bshape[1]);
        span = 128;
        strides[0] = stride_or(op.kdim, op.ld);
        span = std::max<uint64_t>(span, strides[0] * dims[1]);
        strides[1] = 128;
        strides[2] = stride_or(op.bshape[2], op.bstride[2]);
        span = std::max<uint64_t>(span, strides[2] * dims[3]);
        strides[3] = stride_or(op.bshape[1], op.bstride[1]);
        box[0] = 32;
        box[1] = static_cast<cuuint32_t>(bk);
        box[2] = static_cast<cuuint32_t>(box_rows / 32);
        if (encode(map, op.ptr, dims, strides, box, mn_swz) == CUDA_SUCCESS) {
            *mode = kMnSingleBox;
            return MNI_B200_OK;
        }
        box[2] = 1;   // fall through to the multi-box form
    }
    CUtensorMapSwizzle swz;
    if (op.k_major) {
        dims[0] = static_cast<cuuint64_t>(op.kdim);
        dims[1] = static_cast<cuuint64_t>(op.rows);
        box[0] = static_cast<cuuint32_t>(bk);
        box[1] = static_cast<cuuint32_t>(box_rows);
        swz = bk == 32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
        *mode = kKMajor;
    } else {
        dims[0] = static_cast<cuuint64_t>(op.rows);
        dims[1] = static_cast<cuuint64_t>(op.kdim);
        box[0] = 32;
        box[1] = static_cast<cuuint32_t>(bk);
        swz = mn_swz;
        *mode = kMnMultiBox;
    }
    span = std::max<uint64_t>(16, (static_cast<uint64_t>(dims[0]) * 4u + 15u) & ~15ull);
    strides[0] = stride_or(static_cast<int64_t>(dims[1]), op.ld);
    span = std::max<uint64_t>(span, strides[0] * dims[1]);
    for (int i = 0; i < 3; ++i) {   // map dim 2 = innermost batch dim
        const int bi = 2 - i;
        dims[2 + i] = static_cast<cuuint64_t>(op.bshape[bi]);
        strides[1 + i] = stride_or(op.bshape[bi], op.bstride[bi]);
        span = std::max<uint64_t>(span, strides[1 + i] * dims[2 + i]);
    }
    const CUresult r = encode(map, op.ptr, dims, strides, box, swz);
    if (r != CUDA_SUCCESS)
        return fail(MNI_B200_ERR_CUDA,
                    "cuTensorMapEncodeTiled failed (%d): dims %llu x %llu, ld %lld, k_major %d", static_cast<int>(r),
                    static_cast<unsigned long long>(dims[0]), static_cast<unsigned long long>(dims[1]),
                    static_cast<long long>(op.ld), static_cast<int>(op.k_major));
    return MNI_B200_OK;
}

// Tensor map of an operand in 16-bit halves.  K-major: (kdim, rows, batch, plane) in boxes of 64 x 128.  MN-major: (64 contiguous
// rows, kdim, chunks of 64 rows, batch, plane) in boxes of 64 x 64 x 2; the pitch is a multiple of 64 there.
int make_half_map(CUtensorMap *map, const HalfOperand &op, int *mode) {
    if (!encode_fn()) return fail(MNI_B200_ERR_CUDA, "cuTensorMapEncodeTiled entry point not found");
    cuuint64_t dims[5], strides[4];
    cuuint32_t box[5] = {64, 128, 1, 1, 1};
    const cuuint64_t pitch = static_cast<cuuint64_t>(op.pitch) * 2, matrix = static_cast<cuuint64_t>(op.matrix) * 2,
                     plane = static_cast<cuuint64_t>(op.plane) * 2, batch = static_cast<cuuint64_t>(op.batch);
    if (op.k_major) {
        dims[0] = static_cast<cuuint64_t>(op.kdim); dims[1] = static_cast<cuuint64_t>(op.rows); dims[2] = batch; dims[3] = static_cast<cuuint64_t>(op.planes); dims[4] = 1;
        strides[0] = pitch; strides[1] = matrix; strides[2] = plane; strides[3] = 2 * plane;
        *mode = kKMajor;
    } else {
        dims[0] = 64; dims[1] = static_cast<cuuint64_t>(op.kdim); dims[2] = static_cast<cuuint64_t>((op.rows + 63) / 64); dims[3] = batch; dims[4] = static_cast<cuuint64_t>(op.planes);
        strides[0] = pitch; strides[1] = 128; strides[2] = matrix; strides[3] = plane;
        box[1] = 64; box[2] = 2;
        *mode = kMnSingleBox;
    }
    const CUresult r = encode(map, op.ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
    if (r != CUDA_SUCCESS) return fail(MNI_B200_ERR_CUDA, "cuTensorMapEncodeTiled(halves) failed (%d)", static_cast<int>(r));
    return MNI_B200_OK;
}

// Tensor map of the output (or of the split-K partial buffer): dims (N, M, batches), 32 x 32 boxes.
int make_output_map(CUtensorMap *map, float *ptr, int64_t N, int64_t M, int64_t batches, int64_t ld, int64_t bstride) {
    cuuint64_t dims[5] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(M), static_cast<cuuint64_t>(batches), 1, 1};
    cuuint64_t strides[4];
    strides[0] = static_cast<cuuint64_t>(M > 1 ? ld * 4 : ((N * 4 + 15) & ~15LL));
    strides[1] = static_cast<cuuint64_t>(batches > 1 ? bstride * 4 : std::max<int64_t>(strides[0] * M, 16));
    strides[2] = strides[1] * static_cast<cuuint64_t>(batches);
    strides[3] = strides[2];
    const cuuint32_t box[5] = {32, 32, 1, 1, 1};
    const CUresult r = encode(map, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (r != CUDA_SUCCESS) return fail(MNI_B200_ERR_CUDA, "cuTensorMapEncodeTiled(output) failed (%d)", static_cast<int>(r));
    return MNI_B200_OK;
}

struct Plan {
    int bn, bk, cg, stages, splits, tiles_m, tiles_n, grid;   // cg = CTAs per tile (1, or 2 = CTA pair)
    int patches;                                              // epilogue staging patches per warp
    bool ta;                                                  // A operand of the MMAs from tensor memory
    bool sk;                                                  // balanced tail: the last, ragged wave is cut by k-blocks
    int sk_first_tile;
    double est_us;                                            // the cost model's time for this plan (0: it has none)
    int tail_ways, tail_tiles;                                // split tail: the last wave's tiles, cut into this many units each (0: none)
    bool running;                                             // units of several pieces are summed in the epilogue's registers
    size_t smem;
};

constexpr size_t kFixedSmemNoEpi = 1024 + kBarBytes;

// Split tail of `tiles` 256-wide pair tiles: the last wave's tiles cut into `ways` units each (1: not), and what the schedule then
// takes, in rounds of whole tiles, and the finish in microseconds.
struct Cut {
    long long ways;
    double rounds, finish_us;
};
constexpr double kPairNs = 30.0;             // main loop of a 256-wide pair, 3xTF32, per contraction element
// Microseconds of a finish kernel that adds `parts` partial results of `bytes` each: its launch and its traffic.
double finish_us(double parts, double bytes) { return 1.5 + (parts + 1.0) * bytes * 1e-6 / 3.0; }

// After at least one whole round, a last wave that fills at most half of the slots, in a schedule that would idle more than a
// fifth of them, is cut into two to four units per tile of at least 128 contraction elements each.  Otherwise, where a round
// takes long, into as many units as even out best over several short rounds, if that saves 6 % and 5 us: 3xTF32 contractions from
// about 3000 on with 0.5 to 0.8 or 1.5 to 1.75 waves of tiles (74 pairs; us whole / balanced tail / cut): 2048 x 4096 x 1280
// 128 / 91 / 92, 2048 x 8192 x 1280 242 / 174 / 176, 1536 x 8192 x 2048 239 / 197 / 191, 2048 x 8192 x 3584 500 / 436 / 439,
// 2048 x 3072 x 3584 177 / 169 / 168; at K = 2048, 121 / 117 / -, it would save 4.6 %.  Not in single-pass mode, whose long units
// lose more by giving up their running sum (2048 x 8192 x 3584 200 / 209 / 231), and not beside another product, which uses the
// SMs that the wave leaves.  `round_only`: neither.
Cut cut_tail(long long tiles, long long slots, long long k, bool round_only) {
    const long long full = tiles / slots, rem = tiles - full * slots;
    const double tile_bytes = 4.0 * 2 * BM * 256;
    const Cut whole{1, static_cast<double>(rem > 0 ? full + 1 : full), 0.0};
    if (rem == 0) return whole;
    const long long ways = std::min<long long>(slots / rem, 4);
    const double eff = static_cast<double>(tiles) / static_cast<double>((full + 1) * slots);
    if (full >= 1 && ways >= 2 && eff < 0.80 && k / ways >= 128)
        return Cut{ways, static_cast<double>(full) + 1.0 / static_cast<double>(ways), finish_us(static_cast<double>(ways), tile_bytes * static_cast<double>(rem))};
    if (round_only) return whole;
    const double round_us = static_cast<double>(k) * kPairNs * 1e-3;
    Cut best = whole;
    for (long long w = 2; w <= 6 && k / w >= 256; ++w) {
        const Cut c{w, static_cast<double>(full) + static_cast<double>((rem * w + slots - 1) / slots) / static_cast<double>(w),
                    finish_us(static_cast<double>(w), tile_bytes * static_cast<double>(rem))};
        if (c.rounds * round_us + c.finish_us < best.rounds * round_us + best.finish_us) best = c;
    }
    const double saved = (whole.rounds - best.rounds) * round_us - best.finish_us;
    return saved > 5.0 && saved > 0.06 * whole.rounds * round_us ? best : whole;
}
// Longest accumulation chain in tensor memory, in k-blocks (MNI_B200_CHUNK_K contraction elements; 0 = no limit).  The fused
// activation needs the whole sum in one accumulator.
constexpr int kHalfChunkK = 4096;
int chunk_iters_for(const GemmProblem &p, int bk) {
    const int chunk_k = env_int("MNI_B200_CHUNK_K", p.ha ? kHalfChunkK : 1024);
    return (chunk_k > 0 && p.D == nullptr) ? std::max(1, chunk_k / bk) : 0;
}

// Main loop of a 256-wide pair over 16-bit planes, nanoseconds per contraction element, in a loop of calls (the pipe's own 12.6
// and 4.2 at 1.9 GHz are out of reach of the power, and of L2, which feeds 32 and 16 KB a pair and 16 elements).
double half_pair_ns(const GemmProblem &p) { return p.fast_tf32 ? 6.5 : 15.0; }

// Longest of the CTA pairs' shares when groups of units of equal cost are dealt out one after the other, round-robin.
struct UnitGroup {
    long long count;
    double cost;
};
double longest_share(const UnitGroup *groups, int n, int slots) {
    auto share = [&](long long s) {
        double load = 0.0;
        long long at = 0;
        for (int i = 0; i < n; ++i) {
            const long long first = (s - at % slots + slots) % slots;       // this slot's first unit of the group
            if (first < groups[i].count) load += static_cast<double>((groups[i].count - 1 - first) / slots + 1) * groups[i].cost;
            at += groups[i].count;
        }
        return load;
    };
    double most = share(0);            // it changes only where a group begins
    long long at = 0;
    for (int i = 0; i < n; ++i) {
        at += groups[i].count;
        most = std::max(most, share(at % slots));
    }
    return most;
}

// Plans for one or two products of 16-bit planes that share a launch: 256-wide pairs throughout, dealt out in the order given.
// Where units are few, the contractions are split (for a finish kernel that adds the parts), or the last tiles are cut, so that
// the pairs' shares even out.  Returns the estimated microseconds.  A unit costs its main loop and what the pipe waits between
// units; a launch 8 us for its first operands and its last stores.
double find_half_plans(const GemmProblem *p, int count, int sm_count, Plan *pl) {
    const int slots = std::max(1, sm_count / 2);
    const bool one = p[0].fast_tf32;
    auto unit_us = [&](double k_us) { return std::max(k_us + (one ? 1.0 : 4.5), 4.5); };     // ... or its stores
    struct {
        long long tiles, iters, chunk;
        double k_us, out_bytes;
    } w[2];
    for (int i = 0; i < count; ++i) {
        Plan &q = pl[i] = Plan{};
        q.bn = 256;
        q.bk = 64;
        q.cg = 2;
        q.patches = 1;
        const size_t stage = static_cast<size_t>(BM + 128) * q.bk * 2, fixed = 1024 + kBarBytes + static_cast<size_t>(kEpiWarps) * kEpiBufBytes;
        q.stages = static_cast<int>(std::min<size_t>(kMaxStages, (227 * 1024 - fixed) / stage));
        q.smem = fixed + static_cast<size_t>(q.stages) * stage;
        q.tiles_m = static_cast<int>((p[i].M + 255) / 256);
        q.tiles_n = static_cast<int>((p[i].N + 255) / 256);
        q.splits = 1;
        w[i].tiles = static_cast<long long>(p[i].batch) * q.tiles_m * q.tiles_n;
        w[i].iters = p[i].fold * ((p[i].K + q.bk - 1) / q.bk);
        w[i].chunk = chunk_iters_for(p[i], q.bk);
        w[i].k_us = static_cast<double>(w[i].iters * q.bk) * half_pair_ns(p[i]) * 1e-3;
        w[i].out_bytes = 4.0 * static_cast<double>(p[i].batch) * static_cast<double>(p[i].M) * static_cast<double>(p[i].N);
    }
    auto pieces = [&](int i, long long splits) { return w[i].chunk > 0 && (w[i].iters + splits - 1) / splits > w[i].chunk + (w[i].chunk >> 3); };
    constexpr int kWays[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32};
    double best = 1e300;
    int best_splits[2] = {1, 1}, best_cut = 1;
    const int last = count - 1;
    for (const int s0 : kWays)
        for (const int s1 : kWays) {
            const int splits[2] = {s0, s1};
            if (count == 1 && s1 > 1) break;
            bool ok = true;
            double finish = 0.0;
            UnitGroup g[3];
            for (int i = 0; i < count; ++i) {
                ok = ok && (splits[i] == 1 || (p[i].D == nullptr && w[i].iters / splits[i] >= 4 && w[i].tiles * splits[i] <= 2 * slots));
                g[i] = UnitGroup{w[i].tiles * splits[i], unit_us(w[i].k_us / splits[i])};
                if (splits[i] > 1) finish += finish_us(splits[i], w[i].out_bytes);
            }
            if (!ok) continue;
            const double t = longest_share(g, count, slots) + finish;
            if (t < best) { best = t; best_splits[0] = s0; best_splits[1] = s1; best_cut = 1; }
            // ... or the tiles of the last product that the last, ragged wave holds, cut; not where a running sum would be given up
            const long long rem = (g[0].count + (count == 2 ? g[1].count : 0)) % slots;
            if (splits[last] > 1 || rem == 0 || rem > w[last].tiles || (one && (pieces(0, s0) || pieces(last, 1)))) continue;
            for (int ways = 2; ways <= 6 && w[last].iters / ways >= 4; ++ways) {
                g[last].count = w[last].tiles - rem;
                g[count] = UnitGroup{rem * ways, unit_us(w[last].k_us / ways)};
                const double c = longest_share(g, count + 1, slots) + finish + finish_us(ways, 4.0 * 2 * BM * 256 * static_cast<double>(rem));
                if (c < 0.97 * best) { best = c; best_splits[0] = s0; best_splits[1] = s1; best_cut = ways; }
            }
        }
    long long units = 0;
    for (int i = 0; i < count; ++i) {
        pl[i].splits = best_splits[i];
        units += w[i].tiles * pl[i].splits;
    }
    if (best_cut > 1) {
        pl[last].tail_ways = best_cut;
        pl[last].tail_tiles = static_cast<int>(units % slots);
        units += static_cast<long long>(pl[last].tail_tiles) * (best_cut - 1);
    }
    for (int i = 0; i < count; ++i) {
        pl[i].grid = static_cast<int>(std::min<long long>(units, slots)) * 2;
        pl[i].running = pieces(i, pl[i].splits);
        pl[i].est_us = 8.0 + best;
    }
    return 8.0 + best;
}

// A call asks several times (the estimate, its scratch, the launch), and a loop of calls the same again: the last few answers are
// kept, a pure function of the sizes.
double make_half_plans(const GemmProblem *p, int count, int sm_count, Plan *pl) {
    struct Entry {
        int64_t key[14];
        Plan pl[2];
        double us;
    };
    static thread_local Entry entries[8];
    static thread_local unsigned next = 0;
    int64_t key[14] = {count, sm_count, chunk_iters_for(p[0], 64), p[0].fast_tf32};
    for (int i = 0; i < count; ++i) {
        const int64_t k[5] = {p[i].M, p[i].N, p[i].K, p[i].batch, p[i].fold * 2 + (p[i].D != nullptr ? 1 : 0)};
        std::copy(k, k + 5, key + 4 + 5 * i);
    }
    for (const Entry &e : entries)
        if (std::equal(key, key + 14, e.key)) {
            std::copy(e.pl, e.pl + count, pl);
            return e.us;
        }
    Entry &e = entries[next++ % 8];
    e.us = find_half_plans(p, count, sm_count, e.pl);
    std::copy(key, key + 14, e.key);
    std::copy(e.pl, e.pl + count, pl);
    return e.us;
}

Plan make_plan(const GemmProblem &p, int sm_count) {
    Plan pl;
    pl.bn = p.N <= 64 ? 64 : (p.N <= 128 ? 128 : 256);
    const int bn_env = env_int("MNI_B200_BN", 0);
    if (bn_env == 64 || bn_env == 128 || bn_env == 256) pl.bn = bn_env;
    // CTA pairs: 256-wide tiles and at least two 128-row blocks of output.
    const int pair_env = env_int("MNI_B200_CTA_PAIR", 1);     // 0 never, 1 for 256-wide tiles, 2 for every width
    auto pair_for = [&](int bn) { return (p.M > BM && (pair_env >= 2 || (pair_env == 1 && bn == 256))) ? 2 : 1; };
    // Problems with fewer 128 x 256 tiles than SMs are latency-bound: one tile's k-loop is a serial
    // TMA -> split -> MMA chain, so narrower tiles and a K split put more SMs on it.  The tile width and the
    // split are chosen by a small cost model fitted to measured times of 256^3 .. 1024^3 products:
    // nanoseconds per k element of one tile (30 / 33 for a 256-wide pair / lone CTA, 15.4 for 128, 13.5
    // for 64), 1.5 us for the reduce launch and its traffic at 3 TB/s.
    int model_splits = 0;
    pl.est_us = 0.0;
    constexpr double kFixedUs = 5.0;                          // launch, pipeline fill, last epilogue
    const long long tiles256 = static_cast<long long>(p.batch) * ((p.M + BM - 1) / BM) * ((p.N + 255) / 256);
    if (bn_env == 0 && p.force_splits <= 0 && tiles256 < sm_count && env_int("MNI_B200_PLAN_MODEL", 1) != 0) {
        const double k_eff = static_cast<double>(p.K) * static_cast<double>(p.fold);
        const double out_bytes = 4.0 * static_cast<double>(p.batch) * static_cast<double>(p.M) * static_cast<double>(p.N);
        double best = 1e300;
        for (int bn : {256, 128, 64}) {
            if (bn > 64 && p.N <= bn / 2) continue;               // no tile wider than the output needs
            const int cg = pair_for(bn);
            const long long tiles = static_cast<long long>(p.batch) * ((p.M + BM * cg - 1) / (BM * cg)) * ((p.N + bn - 1) / bn);
            const long long slots = std::max(1, sm_count / cg);
            for (int sp : {1, 2, 3, 4, 6, 8, 12, 16}) {
                if (sp > 1 && (tiles * sp > slots || k_eff / sp < 64.0)) continue;
                // A 128-wide tile with a long contraction runs at its steady state, which shared-memory bandwidth
                // sets (128 KB per 32-deep k-block = 1000 cycles): measured 20.5 ns per k element at K = 8192,
                // against 32 for a 256-wide pair doing twice the work.
                const double c_ns = bn == 256 ? (cg == 2 ? 30.0 : 33.0) : (bn == 128 ? (k_eff / sp >= 1024.0 ? 20.5 : 15.4) : 13.5);
                const double rounds = static_cast<double>((tiles * sp + slots - 1) / slots);
                const double t = rounds * (k_eff / sp) * c_ns + (sp > 1 ? 1500.0 + (sp + 1) * out_bytes / 3000.0 : 0.0);
                if (t < best) { best = t; pl.bn = bn; model_splits = sp; }
            }
            // ... or a single, partly filled wave of 256-wide pairs cut like a last one
            if (bn == 256 && cg == 2 && !p.exchanged && tiles < slots) {
                const Cut cut = cut_tail(tiles, slots, p.fold * ((p.K + 15) / 16) * 16, p.fast_tf32 || p.beside);
                const double t = cut.rounds * k_eff * kPairNs + cut.finish_us * 1e3;
                if (cut.ways > 1 && t < 0.97 * best) { best = t; pl.bn = bn; model_splits = 1; }
            }
        }
        pl.est_us = best * 1e-3 + kFixedUs;
    }
    // Problems of several rounds: a round costs the main loop of a tile (nanoseconds per k element) plus its own overhead,
    // or the time to write the round's tiles where the contraction is short, half as much again if the output's rows are
    // not 16-byte aligned.  Fitted to products of 64 .. 1024 in every dimension; it decides against 256-wide tiles where
    // they would compute and write mostly padding (48 x [333 x 64 x 333]: 36.5 us in 256-wide pairs, 25.8 in 128-wide tiles).
    if (bn_env == 0 && p.force_splits <= 0 && !p.fast_tf32 && p.N > 128 && tiles256 >= sm_count && env_int("MNI_B200_PLAN_MODEL", 1) != 0) {
        const double k_us = static_cast<double>(p.K) * static_cast<double>(p.fold) * 1e-3;
        const double unaligned = (p.ldc % 4 != 0 || p.c_bstride % 4 != 0) ? 1.45 : 1.0;
        double best = 1e300;
        for (int bn : {256, 128, 64}) {
            const int cg = pair_for(bn);
            const long long tiles = static_cast<long long>(p.batch) * ((p.M + BM * cg - 1) / (BM * cg)) * ((p.N + bn - 1) / bn);
            const long long slots = std::max(1, sm_count / cg);
            const double loop = k_us * (bn == 256 ? (cg == 2 ? kPairNs : 33.0) : (bn == 128 ? 19.0 : 13.0)) + (bn == 256 ? 0.5 : (bn == 128 ? 1.0 : 0.65));
            const double write = unaligned * (bn == 256 ? (cg == 2 ? 3.7 : 4.5) : (bn == 128 ? 2.2 : 1.5));
            double rounds = static_cast<double>((tiles + slots - 1) / slots);
            if (bn == 256 && cg == 2) {
                const Cut cut = cut_tail(tiles, slots, p.fold * ((p.K + 15) / 16) * 16, p.fast_tf32 || p.beside);
                if (cut.ways > 1) rounds = cut.rounds + 0.25;
            }
            const double t = rounds * std::max(loop, write);
            if (t < best) { best = t; pl.bn = bn; }
        }
        pl.est_us = best + kFixedUs;
    }
    pl.cg = pair_for(pl.bn);
    pl.bk = (pl.bn == 256 && !p.fast_tf32) ? 16 : 32;
    const int bk_env = env_int("MNI_B200_BK", 0);
    if ((bk_env == 16 || bk_env == 32) && pl.bn == 256) pl.bk = bk_env;   // narrower tiles are built for BK = 32 only
    // Narrow tiles of a lone CTA are bound by shared-memory bandwidth; taking A from tensor memory removes
    // most of A's share of it.
    pl.ta = !p.fast_tf32 && pl.cg == 1 && pl.bk == 32 && pl.bn <= 128 && env_int("MNI_B200_TMEM_A", 1) != 0;
    const size_t raw = static_cast<size_t>(BM + pl.bn / pl.cg) * pl.bk * 4;
    const size_t stage = p.fast_tf32 ? raw : (pl.ta ? raw + static_cast<size_t>(pl.bn) * pl.bk * 4 : 2 * raw);
    const size_t budget = 227 * 1024;
    pl.patches = env_int("MNI_B200_EPI_PATCHES", 1) == 2 ? 2 : 1;   // staging patches per epilogue warp
    const size_t fixed = kFixedSmemNoEpi + static_cast<size_t>(kEpiWarps * pl.patches) * kEpiBufBytes;
    pl.stages = static_cast<int>(std::min<size_t>(kMaxStages, (budget - fixed) / stage));
    if (pl.ta) pl.stages = std::min(pl.stages, (512 - 2 * pl.bn) / (2 * pl.bk));   // one TMEM slot per stage
    const int st_env = env_int("MNI_B200_STAGES", 0);
    if (st_env >= 1 && st_env <= pl.stages) pl.stages = st_env;
    pl.smem = fixed + static_cast<size_t>(pl.stages) * stage;
    const int tile_m = BM * pl.cg;
    const int slots = std::max(1, sm_count / pl.cg);          // CTAs (or CTA pairs) that run at once
    pl.tiles_m = static_cast<int>((p.M + tile_m - 1) / tile_m);
    pl.tiles_n = static_cast<int>((p.N + pl.bn - 1) / pl.bn);
    const long long tiles = static_cast<long long>(p.batch) * pl.tiles_m * pl.tiles_n;
    const long long iters = p.fold * ((p.K + pl.bk - 1) / pl.bk);
    int splits = 1;
    if (p.force_splits > 0) {
        splits = p.force_splits;
    } else if (model_splits > 0) {
        splits = model_splits;
    } else if (tiles * 2 <= slots && iters >= 8) {
        // Few output tiles and a long contraction: split K so that the whole GPU works.
        splits = static_cast<int>(std::min<long long>(slots / tiles, iters / 4));
    } else if (pl.ta && iters * pl.bk >= 2048) {
        // Narrow tiles in a few long rounds: the contraction split two to four ways where that evens them out by 6 % and 5 us
        // (100 x [384 x 4096 x 64], 300 tiles on 148 SMs: 182 -> 172 us; 200 x [128 x 2048 x 64]: 74 -> 68).
        const double round_us = static_cast<double>(iters * pl.bk) * (pl.bn == 128 ? 20.5e-3 : 16.0e-3);
        const double bytes = 4.0 * static_cast<double>(p.batch) * static_cast<double>(p.M) * static_cast<double>(p.N);
        const double whole = static_cast<double>((tiles + slots - 1) / slots) * round_us;
        double best = std::min(0.94 * whole, whole - 5.0);
        for (int sp = 2; sp <= 4; ++sp) {
            const double t = static_cast<double>((tiles * sp + slots - 1) / slots) / sp * round_us + finish_us(sp, bytes);
            if (t < best) { best = t; splits = sp; }
        }
    }
    splits = static_cast<int>(std::max<long long>(1, std::min<long long>(std::min<long long>(splits, iters), 64)));
    pl.splits = splits;
    const long long units = tiles * splits;
    pl.grid = static_cast<int>(std::min<long long>(units, slots)) * pl.cg;
    // Balanced tail: the k-blocks of the last wave are dealt out evenly (every slot gets one contiguous range; tiles cut by
    // a range boundary are summed in the owner's epilogue, in slot order).
    pl.sk = false;
    pl.sk_first_tile = 0;
    pl.tail_ways = pl.tail_tiles = 0;
    pl.running = false;
    // MNI_B200_STREAMK=1 turns it on where whole tiles would idle more than 8 % of the slot-rounds.  Off by default: where the
    // contraction is short, parking and adding the shared tiles costs more than the idle slots (24 x [512 x 512 x 64] 19.9 us
    // against 12.4, 6 x 700^3 42.1 / 29.0, 3000 x 1000 x 900 45.8 / 37.7), where it is long the cut below is as fast and its
    // accumulation chains are shorter.
    // MNI_B200_STREAMK=0 turns the split tail below off as well.
    const int sk_env = env_int("MNI_B200_STREAMK", -1);
    // The split tail's partial tiles are added by one small kernel.  2048 x 3072, K = 768 (96 tiles on 74 pairs): two
    // rounds 49.7 us, the balanced tail 51.9 (17 of it parking and adding in the last CTAs), this 41.
    // Neither it nor the running sum is built for exchanged operands, whose patches leave transposed (the planner's own
    // choice there is a 64-wide tile; MNI_B200_BN=256 makes it a 256-wide pair).
    if (splits == 1 && sk_env < 0 && p.force_splits <= 0 && pl.cg == 2 && pl.bn == 256 && !p.exchanged) {
        const Cut cut = cut_tail(tiles, slots, iters * pl.bk, p.fast_tf32 || p.beside);
        if (cut.ways > 1) {
            pl.tail_ways = static_cast<int>(cut.ways);
            pl.tail_tiles = static_cast<int>(tiles % slots);
            pl.grid = static_cast<int>(std::min<long long>(tiles + pl.tail_tiles * (cut.ways - 1), slots)) * pl.cg;
            return pl;
        }
    }
    if (splits == 1 && p.D == nullptr && sk_env > 0) {
        const long long full_rounds = tiles / slots, rem = tiles - full_rounds * slots;
        const double eff = static_cast<double>(tiles) / static_cast<double>((full_rounds + 1) * slots);
        if (rem > 0 && eff < 0.92 && iters >= 8 && tiles * 2 > slots) {
            // the tail takes one whole round along when there is one, so that a range is at least a tile long
            const long long whole = full_rounds > 0 ? full_rounds - 1 : 0;
            const long long range = (tiles - whole * slots) * iters / slots;
            // a tile is shared by at most iters / range + 2 units
            // compiled for the variants that meet ragged waves in practice: 256-wide pairs and narrow tensor-memory tiles
            const bool built = (pl.cg == 2 && pl.bn == 256) || pl.ta;
            if (built && range >= 8 && iters / range + 2 <= kSkMaxShare) {
                pl.sk = true;
                pl.sk_first_tile = static_cast<int>(whole * slots);
                pl.grid = static_cast<int>(slots) * pl.cg;
            }
        }
    }
    // Units summed in several pieces (the kernel's first_piece rule) keep their running sum in registers where that is built.
    const long long chunk = chunk_iters_for(p, pl.bk), unit_len = (iters + splits - 1) / splits;
    pl.running = pl.cg == 2 && pl.bn == 256 && pl.bk == (p.fast_tf32 ? 32 : 16) && !pl.sk && !p.exchanged && chunk > 0 &&
                 unit_len > chunk + (chunk >> 3);
    return pl;
}

// N extent of the MMAs.  A lone CTA's tile that is wider than the output multiplies only the columns that exist
// (units of 16 for a 128-row MMA; whole 32-float chunks when B is read MN-major): an MMA's time is proportional
// to its N, and a 64-wide tile over a 16-column output would spend three quarters of the tensor pipe on zeros.
// The rest of the accumulator is never written, and never stored: the epilogue clips at N.
// MNI_B200_MMA_NARROW=0 keeps full-width MMAs.
int mma_n_for(const GemmProblem &p, const Plan &pl) {
    if (pl.cg != 1 || p.N >= pl.bn || env_int("MNI_B200_MMA_NARROW", 1) == 0) return pl.bn;
    const int64_t unit = p.B.k_major ? 16 : 32;
    return static_cast<int>(std::min<int64_t>(pl.bn, std::max<int64_t>(unit, (p.N + unit - 1) / unit * unit)));
}

uint32_t desc_hi_bits(uint32_t sbo_bytes, uint32_t layout_type) {
    // upper word of the shared-memory descriptor: SBO [32,46) | version 1 [46,48) | layout [61,64)
    return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (layout_type << 29);
}

template <int BN, int BK, int MODE, int NS, int CG, bool TA = false, int TAIL = kWholeTiles, int SG = 1>
cudaError_t launch_variant(const Plan &pl, const Product *const *w, int count, cudaStream_t stream) {
    // The shared-memory opt-in is an attribute of the function on ONE device: set once per device of the process
    // (a bit per device ordinal; setting it twice from two threads is harmless).
    static std::atomic<uint64_t> opted_in{0};
    int dev = 0;
    cudaError_t attr = cudaGetDevice(&dev);
    if (attr != cudaSuccess) return attr;
    const uint64_t bit = 1ull << (dev & 63);
    if ((opted_in.load(std::memory_order_acquire) & bit) == 0) {
        attr = cudaFuncSetAttribute(gemm_tc_kernel<BN, BK, MODE, NS, CG, TA, TAIL, SG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    227 * 1024);
        if (attr != cudaSuccess) return attr;
        opted_in.fetch_or(bit, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(pl.grid));
    cfg.blockDim = dim3(gemm_threads(NS, TAIL == kRunningSum));
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = CG;
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = CG == 2 ? 2 : 1;
    Products<product_slots(MODE)> g;
    for (int i = 0; i < product_slots(MODE); ++i) g.s[i] = *w[i < count ? i : 0];
    g.count = count;
    return cudaLaunchKernelEx(&cfg, gemm_tc_kernel<BN, BK, MODE, NS, CG, TA, TAIL, SG>, g);
}

}  // namespace

// Flags of the balanced tail: per (CTA, parking place, epilogue warp) a ready flag, raised after an accumulator
// is parked, and per region of a tail tile a ticket; the unit that reduces a tile clears what it used, so the
// array is all zero between launches.
constexpr int kSkFlagCount = 3 * 256 * kEpiWarps;
constexpr int kSkFlagBanks = 2;            // bank 1 serves the launches a backward call puts on the library's side stream
__device__ unsigned int g_sk_flags[kSkFlagBanks * kSkFlagCount];

unsigned int *sk_flags_ptr() {
    static thread_local int cached_dev = -1;
    static thread_local unsigned int *ptr = nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    if (dev != cached_dev) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_sk_flags) != cudaSuccess) return nullptr;
        ptr = static_cast<unsigned int *>(p);
        cached_dev = dev;
    }
    return ptr;
}

// Role wait counters (diagnostics): cycles summed over CTAs that each role spent blocked.
__device__ unsigned long long g_role_waits[8];

unsigned long long *role_wait_ptr() {
    static thread_local int cached_dev = -1;
    static thread_local unsigned long long *ptr = nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    if (dev != cached_dev) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_role_waits) != cudaSuccess) return nullptr;
        ptr = static_cast<unsigned long long *>(p);
        cached_dev = dev;
    }
    return ptr;
}

int read_role_waits(uint64_t out[8], int reset) {
    unsigned long long *ptr = role_wait_ptr();
    if (!ptr) return fail(MNI_B200_ERR_CUDA, "role wait counters unavailable");
    MNI_CUDA(cudaDeviceSynchronize());
    MNI_CUDA(cudaMemcpy(out, ptr, 8 * sizeof(uint64_t), cudaMemcpyDeviceToHost));
    if (reset) MNI_CUDA(cudaMemset(ptr, 0, 8 * sizeof(uint64_t)));
    return MNI_B200_OK;
}

// The kernel's view of a problem.  An output with few rows and many columns would fill at most half of
// every 128-row MMA; with the operands exchanged the kernel computes C^T in 64-wide tiles instead and its
// epilogue stores the 32 x 32 patches transposed, so C is written in place as before.
GemmProblem kernel_view(const GemmProblem &p, bool *transposed) {
    *transposed = false;
    const bool storable = (reinterpret_cast<uintptr_t>(p.C) & 15) == 0 && p.ldc % 4 == 0 && p.c_bstride % 4 == 0 &&
                          p.N % 4 == 0 && env_int("MNI_B200_NO_TMA_STORE", 0) == 0 && env_int("MNI_B200_EPI_VECTOR", 0) == 0;
    if (p.ha != nullptr || p.D != nullptr || p.M > 64 || p.N < 256 || !storable || env_int("MNI_B200_TRANSPOSE_OUT", 1) == 0) return p;
    GemmProblem q = p;
    std::swap(q.A, q.B);
    std::swap(q.M, q.N);
    q.exchanged = true;
    *transposed = true;
    return q;
}

static bool can_fuse_activation(const GemmProblem &p, const Plan &pl) {
    auto aligned = [&](const float *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
    return pl.splits == 1 && p.ldc % 4 == 0 && p.c_bstride % 4 == 0 && aligned(p.D) && (p.C == nullptr || aligned(p.C)) &&
           env_int("MNI_B200_NO_TMA_STORE", 0) == 0 && env_int("MNI_B200_EPI_VECTOR", 0) == 0;
}

bool gemm_tc_can_fuse_activation(const GemmProblem &p, int sm_count) { return can_fuse_activation(p, make_plan(p, sm_count)); }

static int64_t partial_pitch(int64_t n) { return (n + 3) / 4 * 4; }

static size_t partial_bytes(const GemmProblem &p, const Plan &pl, int64_t out_rows, int64_t out_cols);
size_t gemm_tc_partial_bytes(const GemmProblem &p0, int sm_count) {
    bool transposed = false;
    const GemmProblem p = kernel_view(p0, &transposed);
    return partial_bytes(p, make_plan(p, sm_count), p0.M, p0.N);
}
static size_t partial_bytes(const GemmProblem &p, const Plan &pl, int64_t out_rows, int64_t out_cols) {
    if (pl.sk) return static_cast<size_t>(pl.grid) * 2 * BM * pl.bn * sizeof(float);   // two parked accumulators per CTA
    if (pl.tail_ways) return static_cast<size_t>(pl.tail_tiles) * pl.tail_ways * BM * pl.cg * pl.bn * sizeof(float);
    if (pl.splits <= 1) return 0;
    return static_cast<size_t>(pl.splits) * p.batch * out_rows * partial_pitch(out_cols) * sizeof(float);
}

bool gemm_tc_uses_pairs(const GemmProblem &p, int sm_count) {
    bool transposed = false;
    return make_plan(kernel_view(p, &transposed), sm_count).cg == 2;
}

double gemm_tc_estimate_us(const GemmProblem &p, int sm_count) {
    bool transposed = false;
    return p.fast_tf32 ? 0.0 : make_plan(kernel_view(p, &transposed), sm_count).est_us;
}

double gemm_estimate_us(const GemmProblem &p0, int sm_count) {
    bool transposed = false;
    const GemmProblem p = kernel_view(p0, &transposed);
    const Plan pl = make_plan(p, sm_count);
    if (pl.est_us > 0 && !p.fast_tf32) return pl.est_us;
    const double ns = (p.fast_tf32 ? 13.0 : kPairNs) * (pl.bn == 256 ? 1.0 : (pl.bn == 128 ? 0.65 : 0.45));
    const double k = static_cast<double>(p.K) * static_cast<double>(p.fold);
    const double slots = std::max(1, sm_count / pl.cg), tiles = static_cast<double>(p.batch) * pl.tiles_m * pl.tiles_n;
    const double out = 4.0 * static_cast<double>(p.batch) * static_cast<double>(p.M) * static_cast<double>(p.N);
    double rounds = std::ceil(tiles * pl.splits / slots) / pl.splits, finish = pl.splits > 1 ? finish_us(pl.splits, out) : 0.0;
    if (pl.tail_ways) {
        rounds = std::floor(tiles / slots) + std::ceil(pl.tail_tiles * pl.tail_ways / slots) / pl.tail_ways;
        finish = finish_us(pl.tail_ways, 4.0 * BM * pl.cg * pl.bn * pl.tail_tiles);
    }
    return 5.0 + rounds * std::max(k * ns * 1e-3, pl.bn == 256 ? 3.7 : 1.5) + finish;
}

double gemm_halves_estimate_us(const GemmProblem *p, int count, int sm_count) {
    Plan pl[2];
    return make_half_plans(p, count, sm_count, pl);
}

void gemm_halves_partial_bytes(const GemmProblem *p, int count, int sm_count, size_t *bytes) {
    Plan pl[2];
    make_half_plans(p, count, sm_count, pl);
    for (int i = 0; i < count; ++i) bytes[i] = partial_bytes(p[i], pl[i], p[i].M, p[i].N);
}

static std::string describe_plan(const GemmProblem &p, const Plan &pl, bool transposed, bool halves);
void gemm_halves_describe(const GemmProblem *p, int count, int sm_count, std::string *lines) {
    Plan pl[2];
    make_half_plans(p, count, sm_count, pl);
    for (int i = 0; i < count; ++i) lines[i] = describe_plan(p[i], pl[i], false, true);
}

std::string gemm_tc_describe(const GemmProblem &p0, int sm_count) {
    bool transposed = false;
    const GemmProblem p = kernel_view(p0, &transposed);
    return describe_plan(p, make_plan(p, sm_count), transposed, false);
}
static std::string describe_plan(const GemmProblem &p, const Plan &pl, bool transposed, bool halves) {
    // pieces a whole unit's contraction is summed in (the kernel's first_piece rule)
    const long long iters = p.fold * ((p.K + pl.bk - 1) / pl.bk);
    const long long len = (iters + pl.splits - 1) / pl.splits;
    const long long ci = chunk_iters_for(p, pl.bk);
    const int pieces = (ci > 0 && len > ci + ci / 8) ? static_cast<int>((len + ci - 1) / ci) : 1;
    char buf[320];
    snprintf(buf, sizeof(buf),
             "%s m=%lld n=%lld k=%lld batch=%lld fold=%lld bn=%d bk=%d pair=%d tmem_a=%d stages=%d splits=%d "
             "tail=%d grid=%d exchanged=%d single_pass=%d pieces=%d mma_n=%d tail_ways=%d running=%d",
             halves ? "planes" : "tensor", static_cast<long long>(p.M), static_cast<long long>(p.N), static_cast<long long>(p.K),
             static_cast<long long>(p.batch), static_cast<long long>(p.fold), pl.bn, pl.bk, pl.cg == 2 ? 1 : 0,
             pl.ta ? 1 : 0, pl.stages, pl.splits, pl.sk || pl.tail_ways ? 1 : 0, pl.grid, transposed ? 1 : 0, p.fast_tf32 ? 1 : 0,
             pieces, mma_n_for(p, pl), pl.tail_ways, pl.running ? 1 : 0);
    return buf;
}

namespace {
struct SplitFinish {
    const float *partial;
    float *C;
    int64_t ldc, c_bstride, batch, M, N;
    const float *bias;
    bool accumulate;
    int splits;
};
int launch_split_finish(const SplitFinish &f, int dep_mode, cudaStream_t stream) {
    const long long rows = static_cast<long long>(f.batch) * f.M;
    const int64_t pld = partial_pitch(f.N);
    const bool vec = f.N % 4 == 0 && f.ldc % 4 == 0 && f.c_bstride % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(f.C) | reinterpret_cast<uintptr_t>(f.bias)) & 15) == 0;
    const long long items = rows * (pld / 4);
    const unsigned blocks = static_cast<unsigned>((items + 255) / 256);
    const bool small = items < (1LL << 31) - 256;
    const int acc = f.accumulate ? 1 : 0, m = static_cast<int>(f.M), n = static_cast<int>(f.N);
    cudaError_t e;
    if (small) {
        auto reduce = vec ? splitk_reduce_kernel<true, unsigned, FastDiv> : splitk_reduce_kernel<false, unsigned, FastDiv>;
        e = launch_dependent(reduce, dim3(blocks), dim3(256), 0, stream, f.partial, f.C, f.ldc, f.c_bstride, f.bias, acc, f.splits,
                             rows, make_fastdiv(f.M), make_fastdiv(pld / 4), m, n, dep_mode);
    } else {
        auto reduce = vec ? splitk_reduce_kernel<true, long long, long long> : splitk_reduce_kernel<false, long long, long long>;
        e = launch_dependent(reduce, dim3(blocks), dim3(256), 0, stream, f.partial, f.C, f.ldc, f.c_bstride, f.bias, acc, f.splits,
                             rows, f.M, pld / 4, m, n, dep_mode);
    }
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "splitk_reduce_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("splitk_reduce_kernel");
    return MNI_B200_OK;
}
int launch_tail_finish(const GemmProblem &p, const Plan &pl, const KParams &k, const float *partial, int dep_mode, cudaStream_t stream) {
    const bool vec = p.N % 4 == 0 && p.ldc % 4 == 0 && p.c_bstride % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(p.C) | reinterpret_cast<uintptr_t>(p.D)) & 15) == 0;
    const dim3 grid(static_cast<unsigned>(BM * pl.cg / 4), static_cast<unsigned>(pl.tail_tiles));
    const cudaError_t e = launch_dependent(vec ? tail_finish_kernel<true> : tail_finish_kernel<false>, grid, dim3(256), 0, stream,
                                           partial, p.D, pl.bn, BM * pl.cg, dep_mode, k);
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "tail_finish_kernel launch failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("tail_finish_kernel");
    return MNI_B200_OK;
}
}  // namespace

// Fills in what one product of a launch needs.  oM / oN: the output's extents (p.M / p.N are the kernel's).
static int make_product(const GemmProblem &p, const Plan &pl, bool transposed, int64_t oM, int64_t oN, float *partial, uint32_t *err_word,
                        Product &w) {
    if (p.K <= 0) return fail(MNI_B200_ERR_ARG, "empty contraction reached the tensor-core launcher");
    if (transposed && (pl.tail_ways || pl.running))
        return fail(MNI_B200_ERR_ARG, "internal: a plan that stores no transposed patches for exchanged operands");
    if ((pl.splits > 1 || pl.sk || pl.tail_ways) && partial == nullptr)
        return fail(MNI_B200_ERR_WORKSPACE, "split-K launch without partial storage");

    KParams &k = w.p;
    k = KParams{};
    CUtensorMap &tmA = w.A, &tmB = w.B, &tmC = w.C, &tmD = w.D, &tmP = w.P;
    if (p.D != nullptr && !can_fuse_activation(p, pl))
        return fail(MNI_B200_ERR_ARG, "fused activation requested for a problem that cannot carry it");
    const bool half = p.ha != nullptr;
    int rc = half ? make_half_map(&tmA, *p.ha, &k.a_mode) : make_operand_map(&tmA, p.A, BM, pl.bk, &k.a_mode);
    if (rc) return rc;
    // B rows that exist in a tile wider than the output: with a K-major B (one box of whole rows) only those are
    // loaded, split and multiplied; the shared memory behind them is never read.
    const int mma_n = mma_n_for(p, pl);
    k.b_rows_live = (p.B.k_major && mma_n < pl.bn) ? mma_n : pl.bn / pl.cg;
    rc = half ? make_half_map(&tmB, *p.hb, &k.b_mode) : make_operand_map(&tmB, p.B, k.b_rows_live, pl.bk, &k.b_mode);
    if (rc) return rc;

    // Epilogue: TMA store when the destination rows are 16-byte aligned, plain stores otherwise.
    float *dst = pl.splits > 1 ? partial : p.C;
    const int64_t pld = partial_pitch(oN);
    const int64_t dst_ld = pl.splits > 1 ? pld : p.ldc;
    const int64_t dst_bs = pl.splits > 1 ? oM * pld : p.c_bstride;
    const int64_t dst_batches = pl.splits > 1 ? static_cast<int64_t>(pl.splits) * p.batch : p.batch;
    const bool tma_ok = (reinterpret_cast<uintptr_t>(dst) & 15) == 0 && dst_ld % 4 == 0 && dst_bs % 4 == 0 &&
                        env_int("MNI_B200_NO_TMA_STORE", 0) == 0;
    k.epi_mode = kEpiPlainStores;
    const bool vec_ok = (reinterpret_cast<uintptr_t>(dst) & 31) == 0 && dst_ld % 8 == 0 && dst_bs % 8 == 0;
    if (vec_ok && env_int("MNI_B200_EPI_VECTOR", 0) != 0) {
        k.epi_mode = kEpiVectorStores;
        tmC = tmA;
    } else if (tma_ok && (dst != nullptr || p.D != nullptr)) {
        if (dst != nullptr) {
            rc = make_output_map(&tmC, dst, oN, oM, dst_batches, dst_ld, dst_bs);
            if (rc) return rc;
        } else {
            tmC = tmA;
        }
        k.epi_mode = (p.accumulate && pl.splits == 1) ? kEpiTmaReduce : kEpiTmaStore;
    } else {
        tmC = tmA;   // unused by the plain-store epilogue, but must be a valid object
    }
    tmD = tmC;
    if (p.D != nullptr) {
        rc = make_output_map(&tmD, p.D, p.N, p.M, p.batch, p.ldc, p.c_bstride);
        if (rc) return rc;
        k.act = 1;
        k.store_pre = p.C != nullptr ? 1 : 0;
    }

    tmP = tmC;
    if (pl.tail_ways) {      // partial tiles one after the other, rows of pl.bn floats
        rc = make_output_map(&tmP, partial, pl.bn, BM * pl.cg, static_cast<int64_t>(pl.tail_tiles) * pl.tail_ways, pl.bn,
                             static_cast<int64_t>(BM) * pl.cg * pl.bn);
        if (rc) return rc;
    }

    k.M = static_cast<int>(p.M);
    k.N = static_cast<int>(p.N);
    k.transpose_out = transposed ? 1 : 0;
    k.tiles_m = pl.tiles_m;
    k.tiles_n = pl.tiles_n;
    k.group_m = std::max(1, std::min(pl.tiles_m, env_int("MNI_B200_GROUP_M", 16)));
    k.batch = static_cast<int>(p.batch);
    k.kiters = static_cast<int>((p.K + pl.bk - 1) / pl.bk);
    k.fold = static_cast<int>(p.fold);
    k.splits = pl.splits;
    k.dep_mode = p.dep_mode;
    k.chunk_iters = chunk_iters_for(p, pl.bk);
    k.a_batch = static_cast<int>(p.A.batch);
    k.a_d1 = static_cast<int>(p.A.bshape[1]);
    k.a_d2 = static_cast<int>(p.A.bshape[2]);
    k.b_batch = static_cast<int>(p.B.batch);
    k.b_d1 = static_cast<int>(p.B.bshape[1]);
    k.b_d2 = static_cast<int>(p.B.bshape[2]);
    {
        const int last_gm = k.tiles_m % k.group_m == 0 ? k.group_m : k.tiles_m % k.group_m;
        k.fd_splits = make_fastdiv(k.splits);
        k.fd_per_batch = make_fastdiv(static_cast<long long>(k.tiles_m) * k.tiles_n);
        k.fd_group_sz = make_fastdiv(static_cast<long long>(k.group_m) * k.tiles_n);
        k.fd_group_m = make_fastdiv(k.group_m);
        k.fd_last_gm = make_fastdiv(last_gm);
        k.fd_a_cnt = make_fastdiv(k.a_batch); k.fd_a_d1 = make_fastdiv(k.a_d1); k.fd_a_d2 = make_fastdiv(k.a_d2);
        k.fd_b_cnt = make_fastdiv(k.b_batch); k.fd_b_d1 = make_fastdiv(k.b_d1); k.fd_b_d2 = make_fastdiv(k.b_d2);
    }
    {
        const int tiles = k.batch * k.tiles_m * k.tiles_n;
        k.tail_ways = pl.tail_ways;
        k.fd_ways = make_fastdiv(pl.tail_ways);
        k.tail_unit = pl.tail_ways ? tiles - pl.tail_tiles : 0x7fffffff;
        k.units = pl.tail_ways ? k.tail_unit + pl.tail_tiles * pl.tail_ways : tiles * pl.splits;
    }
    k.stages = pl.stages;
    k.epi_patches = pl.patches;
    k.idesc = (1u << 4) | (2u << 7) | (2u << 10) | (((p.A.k_major || pl.ta) ? 0u : 1u) << 15) |
              ((p.B.k_major ? 0u : 1u) << 16) | (static_cast<uint32_t>(mma_n >> 3) << 17) |
              (static_cast<uint32_t>((BM * pl.cg) >> 4) << 24);
    // K-major tile: rows of BK floats, 8-row groups SBO apart, swizzle span = one row.
    // MN-major tile: 32-float chunks of BK k-rows (LBO apart); the 32-byte-unit swizzle repeats every
    // 4 k-rows (SBO = 512), and one 8-deep k-step spans two such groups (1024 bytes).
    const uint32_t k_layout = pl.bk == 32 ? 2u : 4u;   // SWIZZLE_128B : SWIZZLE_64B
    const uint32_t k_sbo = static_cast<uint32_t>(8 * pl.bk * 4);
    const uint32_t mn_lbo = static_cast<uint32_t>(pl.bk * 128);
    const uint32_t mn_sbo = 512, mn_layout = 1;        // SWIZZLE_128B_BASE32B
    if (p.A.k_major) { k.a_desc_hi = desc_hi_bits(k_sbo, k_layout); k.a_desc_lbo = 0; k.a_kstep = 2; }
    else { k.a_desc_hi = desc_hi_bits(mn_sbo, mn_layout); k.a_desc_lbo = ((mn_lbo >> 4) & 0x3FFFu) << 16; k.a_kstep = 64; }
    if (p.B.k_major) { k.b_desc_hi = desc_hi_bits(k_sbo, k_layout); k.b_desc_lbo = 0; k.b_kstep = 2; }
    else { k.b_desc_hi = desc_hi_bits(mn_sbo, mn_layout); k.b_desc_lbo = ((mn_lbo >> 4) & 0x3FFFu) << 16; k.b_kstep = 64; }
    if (half) {
        // kind::f16: f16 operands, 16-deep k-steps.  K-major rows of 64 elements, one swizzle span (k-step 32 bytes); MN-major chunks
        // of 64 rows, LBO apart, of 64 k-lines in groups of 8 (k-step two groups).
        const uint32_t hi = desc_hi_bits(1024, 2), lbo = static_cast<uint32_t>((pl.bk * 128) >> 4) << 16;
        k.idesc = (1u << 4) | ((p.ha->k_major ? 0u : 1u) << 15) | ((p.hb->k_major ? 0u : 1u) << 16) | (32u << 17) | (16u << 24);
        k.a_desc_hi = k.b_desc_hi = hi;
        k.a_desc_lbo = p.ha->k_major ? 0 : lbo;
        k.b_desc_lbo = p.hb->k_major ? 0 : lbo;
        k.a_kstep = p.ha->k_major ? 2 : 128;
        k.b_kstep = p.hb->k_major ? 2 : 128;
        k.b_rows_live = 128;
        k.a_batch = static_cast<int>(p.ha->batch); k.a_d1 = 1; k.a_d2 = k.a_batch;
        k.b_batch = static_cast<int>(p.hb->batch); k.b_d1 = 1; k.b_d2 = k.b_batch;
        k.fd_a_cnt = make_fastdiv(k.a_batch); k.fd_a_d1 = make_fastdiv(1); k.fd_a_d2 = make_fastdiv(k.a_d2);
        k.fd_b_cnt = make_fastdiv(k.b_batch); k.fd_b_d1 = make_fastdiv(1); k.fd_b_d2 = make_fastdiv(k.b_d2);
        k.a_exp = p.ha->exp;
        k.b_exp = p.hb->exp;
        k.half_status = p.half_status;
    }
    k.C = p.C;
    k.ldc = p.ldc;
    k.c_bstride = p.c_bstride;
    k.partial = partial;
    k.partial_ld = pld;
    k.bias = p.bias;
    k.accumulate = p.accumulate;
    k.err = err_word;
    {
        // Tests shorten the limit of the device-side waits; the withhold hook (a stage that never fills, so
        // that the waits do run out) is honoured only together with a limit of at most ~0.1 s.
        const char *w = env_value("MNI_B200_WAIT_CYCLES");
        const long long wc = w ? atoll(w) : 0;
        k.wait_cycles = wc > 0 ? wc : kWaitCycles;
        k.withhold_at = k.wait_cycles <= 200000000LL ? env_int("MNI_B200_TEST_WITHHOLD_KBLOCK", 0) : 0;
    }
    k.prof = env_int("MNI_B200_ROLE_WAITS", 0) ? role_wait_ptr() : nullptr;
    k.sk = pl.sk ? 1 : 0;
    k.sk_first_tile = pl.sk_first_tile;
    k.sk_partial = pl.sk ? partial : nullptr;
    k.sk_flags = nullptr;
    if (pl.sk) {
        k.sk_flags = sk_flags_ptr();
        if (!k.sk_flags) return fail(MNI_B200_ERR_CUDA, "balanced-tail flags unavailable");
        k.sk_flags += (p.flag_bank > 0 ? 1 : 0) * kSkFlagCount;
        // ready flags for 2 parking places per CTA, then one ticket per region of a tail tile (fewer tiles than CTAs)
        if (pl.grid * 3 * kEpiWarps > kSkFlagCount) return fail(MNI_B200_ERR_CUDA, "balanced-tail flag array too small");
    }

    return MNI_B200_OK;
}
static int launch_finish(const GemmProblem &p, const Plan &pl, const KParams &k, float *partial, int64_t oM, int64_t oN, cudaStream_t stream,
                         GemmFinish *defer) {
    if (pl.tail_ways) {
        if (!defer) return launch_tail_finish(p, pl, k, partial, 0, stream);
        *defer = [p, pl, k, partial](int dep_mode, cudaStream_t st) { return launch_tail_finish(p, pl, k, partial, dep_mode, st); };
    } else if (pl.splits > 1) {
        const SplitFinish f{partial, p.C, p.ldc, p.c_bstride, p.batch, oM, oN, p.bias, p.accumulate, pl.splits};
        if (!defer) return launch_split_finish(f, 0, stream);
        *defer = [f](int dep_mode, cudaStream_t st) { return launch_split_finish(f, dep_mode, st); };
    }
    return MNI_B200_OK;
}

int launch_gemm_halves(const GemmProblem *p, int count, float *const *partial, uint32_t *err_word, int sm_count, cudaStream_t stream) {
    Plan pls[2];
    make_half_plans(p, count, sm_count, pls);
    Product w[2];
    const Product *products[2] = {&w[0], &w[count - 1]};
    bool cut = false, running = false, tma = true;
    for (int i = 0; i < count; ++i) {
        const int rc = make_product(p[i], pls[i], false, p[i].M, p[i].N, partial[i], err_word, w[i]);
        if (rc) return rc;
        cut = cut || pls[i].tail_ways > 0;
        running = running || pls[i].running;
        tma = tma && (w[i].p.epi_mode == kEpiTmaStore || w[i].p.epi_mode == kEpiTmaReduce) && p[i].D == nullptr;
    }
    const Plan &pl = pls[0];
    cudaError_t e;
    if (!p[0].fast_tf32) {
        e = cut ? launch_variant<256, 64, kHalfThree, 2, 2, false, kCutTiles>(pl, products, count, stream)
                : launch_variant<256, 64, kHalfThree, 2, 2>(pl, products, count, stream);
    } else if (cut) {
        e = launch_variant<256, 64, kHalfOne, 4, 2, false, kCutTiles>(pl, products, count, stream);
    } else {
        e = running && tma ? launch_variant<256, 64, kHalfOne, 4, 2, false, kRunningSum>(pl, products, count, stream)
                           : launch_variant<256, 64, kHalfOne, 4, 2>(pl, products, count, stream);
    }
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "gemm_tc_kernel set-up failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("gemm_tc_kernel");
    GemmFinish finish[2];
    for (int i = 0; i < count; ++i) {
        const int rc = launch_finish(p[i], pls[i], w[i].p, partial[i], p[i].M, p[i].N, stream, &finish[i]);
        if (rc) return rc;
    }
    const bool both = finish[0] && finish[1];
    for (int i = 0; i < count; ++i) {
        const int rc = finish[i] ? finish[i](both ? i + 1 : 0, stream) : static_cast<int>(MNI_B200_OK);
        if (rc) return rc;
    }
    return MNI_B200_OK;
}

int launch_gemm_tc(const GemmProblem &p0, float *partial, uint32_t *err_word, int sm_count,
                   cudaStream_t stream, GemmFinish *defer) {
    if (p0.M <= 0 || p0.N <= 0 || p0.batch <= 0) return MNI_B200_OK;
    bool transposed = false;
    const GemmProblem p = kernel_view(p0, &transposed);       // p.M / p.N are the kernel's; oM / oN the output's
    const int64_t oM = p0.M, oN = p0.N;
    const Plan pl = make_plan(p, sm_count);
    Product w;
    const int rc = make_product(p, pl, transposed, oM, oN, partial, err_word, w);
    if (rc) return rc;
    const KParams &k = w.p;
    const Product *const products[1] = {&w};
    constexpr int count = 1;
    // Two split groups pay when the k-loop is long enough for the second k-block in flight to matter (measured:
    // K = 512 per unit 33.6 -> 32.8 us per attention-shaped product, 128 k-blocks 57.9 -> 54.4 us; four k-blocks per
    // unit are no faster).  MNI_B200_SPLIT_GROUPS=1/2 forces either.
    int split_groups = 1;
    if (pl.ta) {
        const long long unit_iters = (static_cast<long long>(k.fold) * k.kiters + pl.splits - 1) / pl.splits;
        const int sg_env = env_int("MNI_B200_SPLIT_GROUPS", 0);
        split_groups = (sg_env == 1 || sg_env == 2) ? sg_env : (unit_iters >= 12 ? 2 : 1);
    }
    const bool running = pl.running && (k.epi_mode == kEpiTmaStore || k.epi_mode == kEpiTmaReduce);
    cudaError_t e = cudaErrorInvalidValue;
    if (pl.sk) {
        if (pl.ta && pl.bn == 64 && split_groups == 2) e = launch_variant<64, 32, kThreePass, 8, 1, true, kBalanced, 2>(pl, products, count, stream);
        else if (pl.ta && pl.bn == 64) e = launch_variant<64, 32, kThreePass, 8, 1, true, kBalanced>(pl, products, count, stream);
        else if (pl.ta && pl.bn == 128 && split_groups == 2) e = launch_variant<128, 32, kThreePass, 8, 1, true, kBalanced, 2>(pl, products, count, stream);
        else if (pl.ta && pl.bn == 128) e = launch_variant<128, 32, kThreePass, 8, 1, true, kBalanced>(pl, products, count, stream);
        else if (!p.fast_tf32 && pl.bk == 16) e = launch_variant<256, 16, kThreePass, 8, 2, false, kBalanced>(pl, products, count, stream);
        else if (!p.fast_tf32 && pl.bk == 32) e = launch_variant<256, 32, kThreePass, 8, 2, false, kBalanced>(pl, products, count, stream);
        else if (pl.bk == 16) e = launch_variant<256, 16, kOnePass, 4, 2, false, kBalanced>(pl, products, count, stream);
        else e = launch_variant<256, 32, kOnePass, 4, 2, false, kBalanced>(pl, products, count, stream);
    } else if (running && p.fast_tf32) {
        e = launch_variant<256, 32, kOnePass, 4, 2, false, kRunningSum>(pl, products, count, stream);
    } else if (running) {
        e = launch_variant<256, 16, kThreePass, 8, 2, false, kRunningSum>(pl, products, count, stream);
    } else if (pl.tail_ways) {
        if (!p.fast_tf32 && pl.bk == 16) e = launch_variant<256, 16, kThreePass, 8, 2, false, kCutTiles>(pl, products, count, stream);
        else if (!p.fast_tf32) e = launch_variant<256, 32, kThreePass, 8, 2, false, kCutTiles>(pl, products, count, stream);
        else if (pl.bk == 16) e = launch_variant<256, 16, kOnePass, 4, 2, false, kCutTiles>(pl, products, count, stream);
        else e = launch_variant<256, 32, kOnePass, 4, 2, false, kCutTiles>(pl, products, count, stream);
    } else if (pl.ta) {
        if (pl.bn == 64 && split_groups == 2) e = launch_variant<64, 32, kThreePass, 8, 1, true, kWholeTiles, 2>(pl, products, count, stream);
        else if (pl.bn == 64) e = launch_variant<64, 32, kThreePass, 8, 1, true>(pl, products, count, stream);
        else if (split_groups == 2) e = launch_variant<128, 32, kThreePass, 8, 1, true, kWholeTiles, 2>(pl, products, count, stream);
        else e = launch_variant<128, 32, kThreePass, 8, 1, true>(pl, products, count, stream);
    }
#define MNI_VARIANT(BN_, BK_)                                                                         \
    if (pl.cg == 1 && !pl.ta && pl.bn == BN_ && pl.bk == BK_) {                                                 \
        if (p.fast_tf32) e = launch_variant<BN_, BK_, kOnePass, 4, 1>(pl, products, count, stream);      \
        else e = launch_variant<BN_, BK_, kThreePass, 8, 1>(pl, products, count, stream);                 \
    }
#define MNI_PAIR_VARIANT(BN_, BK_)                                                                    \
    if (pl.cg == 2 && !pl.sk && !pl.tail_ways && !running && pl.bn == BN_ && pl.bk == BK_) {                                                 \
        if (p.fast_tf32) e = launch_variant<BN_, BK_, kOnePass, 4, 2>(pl, products, count, stream);      \
        else e = launch_variant<BN_, BK_, kThreePass, 8, 2>(pl, products, count, stream);                 \
    }
    MNI_PAIR_VARIANT(64, 32) MNI_PAIR_VARIANT(128, 32) MNI_PAIR_VARIANT(256, 16) MNI_PAIR_VARIANT(256, 32)
#undef MNI_PAIR_VARIANT
    MNI_VARIANT(64, 32) MNI_VARIANT(128, 32) MNI_VARIANT(256, 16) MNI_VARIANT(256, 32)
#undef MNI_VARIANT
    if (e != cudaSuccess) return fail(MNI_B200_ERR_CUDA, "gemm_tc_kernel set-up failed: %s", cudaGetErrorString(e));
    MNI_LAUNCH_CHECK("gemm_tc_kernel");
    return launch_finish(p, pl, k, partial, oM, oN, stream, defer);
}

}  // namespace mni
