// FP64-accurate tall-skinny products on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory), for the mixed-precision GCG:
// the Gram products Q^T P and the linear combinations Y = alpha X C + Y
// diag(beta) that the reference computes with DenseMatQtAP and
// MultiVecLinearComb (app/app_lapack.c:64-183, :463-534).
//
// Method (error-free digit splitting, the Ozaki scheme), as in ozaki.cu:
// within an exponent window of consecutive k every row of the left operand
// and every column of the right operand gets an exponent e with |x| < 2^e,
// |x| becomes the 55-bit fixed-point integer X = |x| 2^(55-e) (truncated),
// written as 7 digits of 8 bits with x's sign: the leading digit in [0, 128],
// the others balanced in [-128, 127].  Digits are exact in FP16, the 28 digit
// pairs with i + j <= 6 are multiplied on the tensor cores and summed into 7
// level accumulators L_l = sum_{i+j=l} d_i d'_j, which are exact FP32 integers
// as long as |L_l| < 2^24: 128 consecutive k (|L_6| <= 128 * 7 * 128^2 <
// 2^23.81).  Every 128 k ("chunk") the levels are read out of tensor memory
// into one exact 96-bit integer per output; at the end of a window it is
// converted to FP64 (integer instructions, round to nearest) with the window's
// scale.  A Gram work item has one window over its whole k range (error below
// 2^-53 sqrt(K) |x| |y| per entry, under the FP64 dot product's bound
// K 2^-53 |x| |y|); a linear combination has one per 432 k.
//
// Data path, per CTA (one per SM, persistent over work items, 16 warps):
//  * exponent fields come from a streaming pre-pass (k_tc_expcols /
//    k_tc_exprows: per column of the Gram operands over each window, per row
//    of the linear combination's left operand);
//  * bulk tensor copies (cp.async.bulk.tensor.2d, TMA) bring the raw FP64
//    values of each 32-k stage into shared memory ahead of their use, in boxes
//    with the 128-byte swizzle, so that the lanes of a warp hit distinct banks;
//    the right operand of a linear combination is prepared once per call
//    (k_tc_bprep) and copied into the digit stages with cp.async.bulk;
//  * 16 worker warps turn core matrices (8 rows x 8 k) into the 7 FP16 digit
//    planes of a digit stage (a ring of two, K-major core-matrix layout);
//  * one warp issues the MMAs of each digit stage (M = 128 rows, N = up to
//    256, K = 16, f16 x f16 -> f32 into the 7 level accumulators, 7 x BN of
//    the 512 tensor-memory columns, two sets of them where they fit) and
//    commits them to mbarriers;
//  * every worker drains its slice of the levels after each chunk (warp w reads
//    lanes 32 (w % 4) .. + 31, BN / 4 columns) and folds it at the end of each
//    window (a Gram work item longer than one window adds its windows into its
//    split-k partial).
// Every wait on an mbarrier is bounded; a wait that runs out sets the error
// word and every warp stops at its next wait, so the kernel always returns.
//
// Measured, with the pre-pass (n = 262144; 16-k digit stages, 144-k chunks and
// 128-row tiles before -> now): Gram 100 x 20 223 -> 177 us, 180 x 20 408 -> 305,
// 180 x 40 450 -> 391; linear combination 180 -> 20 352 -> 317 us, 180 -> 40 401 ->
// 366; n = 2097152: Gram 360 x 40 5.11 -> 4.65 ms, 360 -> 40 4.85 -> 4.52, 400 ->
// 320 30.7 -> 28.7.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace gcge {
namespace {

constexpr int kTcDigits = 7;
constexpr int kTcM = 128;      // output rows per tile (tensor-memory lanes)
constexpr int kTcStageK = 32;  // k per stage: two MMA steps
constexpr int kTcDrainStages = 4;
constexpr int kTcDrainK = kTcStageK * kTcDrainStages;  // 128: exact FP32 level sums
constexpr int kTcKGroups = kTcStageK / 8;              // core matrices along k per stage
constexpr int kTcDigStages = 2;                         // ring of digit stages
constexpr int kTcWarps = 16;  // worker warps: digit conversion and drain
constexpr int kTcThreads = (kTcWarps + 1) * 32;  // and one warp issuing the MMAs
constexpr uint32_t kTcTmemCols = 512;
// bounded mbarrier waits: 4 s of device clock, or this many suspended tests
constexpr unsigned long long kTcWaitNs = 4000000000ull;
constexpr long long kTcWaitPolls = 1LL << 22;
// A Gram work item shares one exponent per column over its whole k range
// (at most this many rows: the 96-bit level sums stay below 2^86)
constexpr int kTcSuperGramMax = 16384 * kTcDrainK;
constexpr int kTcSuperLincomb = 432;  // K up to 432 in one window

// Byte layout of one operand tile of R rows in a digit stage: plane i
// (digit), k-group g (8 consecutive k), row r: i * plane + g * lbo +
// (r / 8) * 128 + (r % 8) * 16, with lbo = R * 16 + 16 (the pad keeps the
// 16-byte core-matrix rows of different k-groups on different banks).
__host__ __device__ constexpr uint32_t tc_lbo(int rows) { return (uint32_t)rows * 16u + 16u; }
__host__ __device__ constexpr uint32_t tc_plane(int rows) { return kTcKGroups * tc_lbo(rows); }
__host__ __device__ constexpr uint32_t tc_tile_bytes(int rows) {
    return kTcDigits * tc_plane(rows);
}
__host__ __device__ constexpr uint32_t tc_round(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }
// The right operand's 7 digit planes form ONE tile of 7 BN rows (plane j at
// rows [j BN, (j + 1) BN)), so that a single MMA with N = (7 - i) BN
// multiplies left plane i by right planes 0 .. 6 - i and adds each product
// into its level's accumulator columns (level l = i + j at columns l BN):
// k-group g, row r at g * lbo_b + (r / 8) * 128 + (r % 8) * 16.
__host__ __device__ constexpr uint32_t tc_lbo_b(int bn) {
    return (uint32_t)kTcDigits * bn * 16u + 16u;
}
__host__ __device__ constexpr uint32_t tc_tile_b_bytes(int bn) { return kTcKGroups * tc_lbo_b(bn); }

// Shared memory (offsets from a 1024-byte aligned base).  Raw values arrive in
// boxes with the 128-byte swizzle: of a Gram in halves of a stage (16 k), A
// [rows][16 k] and B [BN rows][16 k], four halves where they fit, else three; of
// a linear combination two halves at once, A [8][32 k][16 rows] (the right
// operand's prepared digit planes are copied straight into the digit stage).
template <int BN, bool GRAM>
struct TcLayout {
    static constexpr uint32_t a_bytes = tc_tile_bytes(kTcM);
    static constexpr uint32_t b_bytes = tc_tile_b_bytes(BN);
    static constexpr uint32_t a_box = 16u * kTcM * 8u;
    static constexpr uint32_t b_box = GRAM ? 16u * BN * 8u : 0u;
    static constexpr uint32_t half_bytes = a_box + b_box;
    static constexpr uint32_t stage_bytes = a_bytes + b_bytes;
    static constexpr uint32_t limit = 232448 - 1024 - 256;  // per CTA, alignment, barriers
    static constexpr int halves =
        4 * half_bytes + kTcDigStages * stage_bytes + 1024 <= limit ? 4 : 3;
    static constexpr uint32_t raw_off = 0;
    static constexpr uint32_t dig_off = tc_round(raw_off + halves * half_bytes, 1024);
    static constexpr uint32_t bar_off = tc_round(dig_off + kTcDigStages * stage_bytes, 16);
    // accumulator sets in tensor memory: two let a chunk be drained while the
    // next one's MMAs run
    static constexpr int accs = 2 * kTcDigits * BN <= (int)kTcTmemCols ? 2 : 1;
    // mbarriers empty[2] full[2] rfull[4] accf[2] fin
    static constexpr int nbars = 2 * kTcDigStages + 7;
    // tmem slot, abort flag, readers' arrivals, raw halves and planes issued
    static constexpr uint32_t misc_off = bar_off + nbars * 8;
    static constexpr uint32_t bytes = misc_off + 48;
    static constexpr uint32_t alloc_bytes = bytes + 1024;  // room to align the base
    static_assert(half_bytes % 1024 == 0, "swizzled boxes start on 1024 bytes");
    static_assert(alloc_bytes <= 232448, "shared memory beyond the per-CTA limit");
};

struct TcArgs {
    int M, N, K;
    const double *A;  // gram: Q (k, r) at A[k + r lda]; lincomb: X (r, k) at A[r + k lda]
    size_t lda;
    int super_k;      // k per exponent window (gram: a multiple of kTcStageK)
    int kchunk;       // gram: k per work item (multiple of super_k)
    int items;        // work items
    int mtiles, ntiles;
    int mrows;        // rows of a tile: a multiple of 8, at most kTcM
    double *out;      // gram: partials [kz][M x N]; lincomb: Y (ldo)
    size_t ldo;
    const double *beta;
    int incb;
    double alpha;
    // exponent fields: gram: eA [window][M], eB [window][N]; lincomb: eA
    // [window][M] (rows of X), eB = the prepared right operand's [ntile][window][BN]
    const int *eA, *eB;
    const uint8_t *bplanes;  // lincomb: [ntile][digit stage][b_bytes]
    int nstages, nsup;       // lincomb: digit stages and exponent windows of K
    int accumulate;          // lincomb: add to Y (later blocks of a split contraction)
    int *error;
};

__device__ __forceinline__ uint32_t su32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// ---------------------------------------------------------------- mbarriers
__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *b, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return done != 0;
}
// The same test, suspending the thread in hardware until the phase completes
// or about `hint_ns` have passed, so that a waiting warp takes no issue slots
// from the warps doing the work.
__device__ __forceinline__ bool mbar_test_suspend(uint64_t *b, uint32_t parity, uint32_t hint_ns) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(su32(b)), "r"(parity), "r"(hint_ns)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ unsigned long long tc_global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Waits for the phase of `parity` to complete; false when the wait ran out
// (kTcWaitNs on the device clock, or kTcWaitPolls tests) or another role
// gave up (abort flag set).  All lanes of the calling warp must call it
// together; lane 0 waits and the result is broadcast.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *b, uint32_t parity,
                                               volatile int *abort_flag, int *gerror) {
    if (__all_sync(0xffffffffu, mbar_test(b, parity))) return true;
    int ok = 1;
    if ((threadIdx.x & 31) == 0 && !mbar_test(b, parity)) {
        const unsigned long long t0 = tc_global_ns();
        long long polls = 0;
        while (!mbar_test_suspend(b, parity, 20000u)) {
            if (*abort_flag) {
                ok = 0;
                break;
            }
            if (++polls > kTcWaitPolls || tc_global_ns() - t0 > kTcWaitNs) {
                *abort_flag = 1;
                atomicExch(gerror, 1);
                ok = 0;
                break;
            }
        }
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    // every lane takes the phase's acquire itself (the phase cannot move on
    // without this warp, so the test succeeds at once)
    if (ok) mbar_test(b, parity);
    return ok != 0;
}

// Arrival on a shared-memory counter (release and acquire at CTA scope);
// returns the count before it.
__device__ __forceinline__ uint32_t smem_arrive(uint32_t *ctr) {
    uint32_t old;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "r"(su32(ctr))
                 : "memory");
    return old;
}

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    // start address, leading (k-direction) and stride (8-row) byte offsets in
    // 16-byte units, descriptor version 1, no swizzle
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
           ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// kind::f16 instruction descriptor: f32 accumulate (bit 4), f16 A and B
// (format 0 at bits 7 and 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t tc_idesc(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t *b) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            su32(b))
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
__device__ __forceinline__ void tc_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One lane of the (converged) calling warp; the compiler then knows the branch
// to be taken by one thread and keeps the MMAs' operands in uniform registers.
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(p));
    return p != 0;
}

// ---------------------------------------------------------------- digits
__device__ __forceinline__ int tc_exp_field(double x) {
    return max((int)(((unsigned)__double2hiint(x) >> 20) & 0x7FFu), 1);
}

// X = |x| 2^(1077 - emax) as a 55-bit fixed-point integer (truncated; the
// caller guarantees emax >= the exponent field of x), plus 0x808080808080,
// as two words: the 53-bit significand at the top of 64 bits, shifted right by
// 9 + emax - field (a 64-bit shift of 64 or more gives 0).  hi = x's high word
// (its sign bit is the sign).
__device__ __forceinline__ void tc_fixed55(double x, uint32_t emax, uint32_t &yh, uint32_t &yl,
                                           uint32_t &hi) {
    hi = (uint32_t)__double2hiint(x);
    const uint32_t lo = (uint32_t)__double2loint(x);
    const uint32_t eb = hi & 0x7FF00000u;  // exponent field << 20
    // the hidden bit, absent for zeros and subnormals (which count as field 1)
    const uint32_t mhi = (hi & 0x000FFFFFu) | min(eb, 0x00100000u);
    const uint32_t xh = __funnelshift_l(lo, mhi, 11);
    const uint32_t field = max(eb, 0x00100000u) >> 20;
    uint32_t sl, sh;
    asm("{\n.reg .b64 t;\nmov.b64 t, {%2, %3};\nshr.u64 t, t, %4;\nmov.b64 {%0, %1}, t;\n}\n"
        : "=r"(sl), "=r"(sh)
        : "r"(lo << 11), "r"(xh), "r"(emax + 9u - field));
    asm("add.cc.u32 %0, %2, 0x80808080;\n\taddc.u32 %1, %3, 0x8080;"
        : "=r"(yl), "=r"(yh)
        : "r"(sl), "r"(sh));
}

// (a - b) on two packed FP16 values
__device__ __forceinline__ uint32_t tc_hsub2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// The 7 FP16 digits of 8 values (one row, 8 consecutive k) relative to the
// exponent field emax: out[i] holds digit i of the 8 values, two per word
// (lower k in the low half).  With Y = X + 0x808080808080 (tc_fixed55),
// digit 0 is Y >> 48 (in [0, 128]) and digit i >= 1 is byte 6 - i of Y less
// 128 (in [-128, 127]), so that X = sum_i d_i 2^(8 (6 - i)); each carries x's
// sign.  A digit is formed for two values at once: the FP16 pattern
// sign | 0x6400 | field is +-(1024 + field) exactly (ulp 1 on [1024, 2048)),
// and subtracting +-1024 (digit 0) or +-(1024 + 128) leaves +-d exactly.
__device__ __forceinline__ void tc_digit_pair(double x0, double x1, uint32_t emax,
                                              uint32_t (&w)[kTcDigits]) {
    uint32_t yh0, yl0, h0, yh1, yl1, h1;
    tc_fixed55(x0, emax, yh0, yl0, h0);
    tc_fixed55(x1, emax, yh1, yl1, h1);
    // +-1024 in each half: the sign bits of the two values at bits 15 and 31
    const uint32_t M = (__byte_perm(h0, h1, 0x7030) & 0x80008000u) | 0x64006400u;
    const uint32_t Mb = M | 0x00800080u;                // +-(1024 + 128)
    w[0] = tc_hsub2(__byte_perm(yh0, yh1, 0x7632) | M, M);
    // byte 6 - i of Y: bytes 4, 5 in the high word, 0..3 in the low word; the
    // permutation puts value 0's byte in half 0 and value 1's in half 1
    w[1] = tc_hsub2((__byte_perm(yh0, yh1, 0x0501) & 0x00FF00FFu) | M, Mb);
    w[2] = tc_hsub2((__byte_perm(yh0, yh1, 0x0400) & 0x00FF00FFu) | M, Mb);
    w[3] = tc_hsub2((__byte_perm(yl0, yl1, 0x0703) & 0x00FF00FFu) | M, Mb);
    w[4] = tc_hsub2((__byte_perm(yl0, yl1, 0x0602) & 0x00FF00FFu) | M, Mb);
    w[5] = tc_hsub2((__byte_perm(yl0, yl1, 0x0501) & 0x00FF00FFu) | M, Mb);
    w[6] = tc_hsub2((__byte_perm(yl0, yl1, 0x0400) & 0x00FF00FFu) | M, Mb);
}
__device__ __forceinline__ void tc_digits8(const double (&v)[8], int emax, uint4 (&out)[kTcDigits]) {
    uint32_t w[4][kTcDigits];
#pragma unroll
    for (int e = 0; e < 4; ++e) tc_digit_pair(v[2 * e], v[2 * e + 1], (uint32_t)emax, w[e]);
#pragma unroll
    for (int i = 0; i < kTcDigits; ++i) out[i] = make_uint4(w[0][i], w[1][i], w[2][i], w[3][i]);
}
// ---------------------------------------------------------------- bulk copies
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(
                     su32(b)),
                 "r"(bytes)
                 : "memory");
}
// contiguous bytes (16-byte aligned, a multiple of 16) into shared memory,
// completing on an mbarrier
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
        "[%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(su32(bar))
        : "memory");
}
// 2D tile of a tensor map into shared memory, completing on an mbarrier
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(su32(bar))
        : "memory");
}


// (vh 2^64 + vl) 2^e as a double, rounded to nearest (ties to even), with
// integer instructions only (FP64 arithmetic is a slow pipe on this part).
// Results below the normal range flush to zero; above it they are +-inf.
__device__ __forceinline__ double tc_i128_f64(long long vh, unsigned long long vl, int e) {
    // vh 2^64 + vl, a two's-complement 128-bit integer
    const bool neg = vh < 0;
    if (neg) {
        vl = ~vl + 1ull;
        vh = ~vh + (vl == 0 ? 1 : 0);
    }
    const unsigned long long mh = (unsigned long long)vh;  // magnitude mh 2^64 + vl
    if ((mh | vl) == 0) return 0.0;
    // the leading 64 bits th (top bit set) and the rest tl
    int lz;
    unsigned long long th, tl;
    if (mh != 0) {
        lz = __clzll((long long)mh);
        th = lz ? (mh << lz) | (vl >> (64 - lz)) : mh;
        tl = vl << lz;
    } else {
        lz = 64 + __clzll((long long)vl);
        th = vl << (lz - 64);
        tl = 0;
    }
    // 53 bits kept, 11 rounded, tl sticky; the magnitude is mant 2^(75 - lz)
    const unsigned long long mant = th >> 11, rb = th & 0x7FFull;
    const bool up = rb > 0x400ull || (rb == 0x400ull && (tl != 0 || (mant & 1ull)));
    const int field = 1023 + 127 - lz + e;
    unsigned long long bits;
    if (field <= 0) {
        bits = 0;
    } else if (field >= 2047) {
        bits = 0x7FF0000000000000ull;
    } else {
        // mant holds the hidden bit, so it adds one to field - 1; a carry of
        // the rounding moves into the exponent
        bits = ((unsigned long long)(field - 1) << 52) + mant + (up ? 1ull : 0ull);
        if (bits > 0x7FF0000000000000ull) bits = 0x7FF0000000000000ull;
    }
    return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}
// A 96-bit two's-complement accumulator (w0 least significant): += (a0, a1, a2)
__device__ __forceinline__ void tc_acc96(uint32_t &w0, uint32_t &w1, uint32_t &w2, uint32_t a0,
                                         uint32_t a1, uint32_t a2) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(w0), "+r"(w1), "+r"(w2)
        : "r"(a0), "r"(a1), "r"(a2));
}

// Waits, with a bound of its own and regardless of the abort flag, for a
// phase that asynchronous work of this CTA still completes (bulk copies or
// MMAs in flight at teardown).  Lane 0 of the calling warp waits.
__device__ __forceinline__ void mbar_wait_teardown(uint64_t *b, uint32_t parity) {
    if ((threadIdx.x & 31) == 0) {
        const unsigned long long t0 = tc_global_ns();
        while (!mbar_test_suspend(b, parity, 20000u))
            if (tc_global_ns() - t0 > 1000000000ull) break;
    }
    __syncwarp();
}

// ---------------------------------------------------------------- work items
// Work item `it`: gram: (m tile, n tile, k range); lincomb: (m tile = 128
// rows of X and Y, n tile).
struct TcItem {
    int mt0, nt, kb, ke;
};
template <bool GRAM>
__device__ __forceinline__ TcItem tc_item(const TcArgs &a, int it) {
    TcItem w;
    const int mn = a.mtiles * a.ntiles;
    const int z = it / mn, r = it % mn;
    w.mt0 = (r % a.mtiles) * a.mrows;
    w.nt = r / a.mtiles;
    if (GRAM) {
        w.kb = z * a.kchunk;
        w.ke = min(a.K, w.kb + a.kchunk);
    } else {
        w.kb = 0;
        w.ke = a.K;
    }
    return w;
}
// Work item it + gridDim.x after w (item it).  A linear combination's items are
// short, so they are stepped instead of divided out.
template <bool GRAM>
__device__ __forceinline__ TcItem tc_item_after(const TcArgs &a, TcItem w, int next) {
    if (GRAM) return tc_item<GRAM>(a, next);
    const int span = a.mtiles * kTcM;
    w.mt0 += (int)gridDim.x * kTcM;
    while (w.mt0 >= span) w.mt0 -= span, ++w.nt;
    return w;
}
// A position in this CTA's sequence of raw stages: work item, window start,
// raw stage start.
struct TcCursor {
    TcItem w;
    int it, sk, k0;
    bool valid;
};
template <bool GRAM>
__device__ __forceinline__ void cur_init(const TcArgs &a, TcCursor &c) {
    c.it = blockIdx.x;
    c.valid = c.it < a.items;
    if (c.valid) {
        c.w = tc_item<GRAM>(a, c.it);
        c.sk = c.k0 = c.w.kb;
    }
}
template <bool GRAM>
__device__ __forceinline__ void cur_next(const TcArgs &a, TcCursor &c) {
    const int ske = min(c.w.ke, c.sk + a.super_k);
    c.k0 += kTcStageK;
    if (c.k0 < ske) return;
    c.sk += a.super_k;
    if (c.sk < c.w.ke) {
        c.k0 = c.sk;
        return;
    }
    c.it += gridDim.x;
    c.valid = c.it < a.items;
    if (c.valid) {
        c.w = tc_item_after<GRAM>(a, c.w, c.it);
        c.sk = c.k0 = c.w.kb;
    }
}

// ---------------------------------------------------------------- kernel
// Warps 0 .. 15 are the workers.  Per stage (32 k) a worker warp converts its
// units, core matrices of 8 rows x 8 k with a pair of consecutive k per lane:
// its share of the left operand's and, for a Gram, its turn of the right
// operand's.  After each drain chunk it moves
// its slice of the level accumulators (tensor-memory lane quarter warp % 4,
// BN / 4 columns) into 96-bit integers, and after an exponent window it folds
// them into FP64.  The last worker to have read a stage's raw halves issues the
// bulk copies that take their buffers.  Warp 16 issues the MMAs of each
// stage once every worker has finished it (a dedicated warp: the issue blocks
// while the tensor core works through the previous stage).
//
// Rows of a tile past the operand's last row group hold whatever the buffers
// held: they reach only output rows (or columns) that are not read.
//
// The workers bound it, by their instructions (half of the issue slots, the ALU
// at 51%) and their latency at four warps per scheduler; the tensor cores are
// busy a quarter of the time, HBM 23% (524288 x 360 x 40, 0.92 ms).  So a stage is as long as shared
// memory allows (a third of the instructions of 16-k stages were waits, cursors
// and addresses), the code is short (a second copy of the conversion cost 5% in
// instruction fetches) and no register is spilled in the loop (the shared memory
// taken leaves no L1: spilled accumulators doubled the time).
//
// The waits form no cycle: stage t is produced after the MMAs of stage t - 2
// completed (a ring of two digit stages); a worker drains chunk c before it
// finishes the first stage of chunk c + accs, whose MMAs overwrite chunk c's
// accumulators.
template <int BN, bool GRAM>
__global__ void __launch_bounds__(kTcThreads, 1)
    k_tc_digits(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                TcArgs a) {
    using L = TcLayout<BN, GRAM>;
    static_assert(BN % 16 == 0 && BN <= 64, "tile width: a multiple of 16, at most 64");
    constexpr int RH = L::halves, ACCS = L::accs;
    // a linear combination's copies take two buffers from an even one on
    static_assert(GRAM || RH == 4, "linear combination: raw buffers in pairs");
    extern __shared__ __align__(1024) uint8_t sm_raw[];
    // 1024-byte aligned base (the 128-byte swizzle of the bulk copies needs it)
    uint8_t *sm = sm_raw + ((1024u - (su32(sm_raw) & 1023u)) & 1023u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + L::bar_off);
    uint64_t *empty = bars, *full = bars + kTcDigStages, *rfull = bars + 2 * kTcDigStages;
    uint64_t *accf = rfull + 4, *fin = rfull + 6;
    uint32_t *misc = reinterpret_cast<uint32_t *>(sm + L::misc_off);
    uint32_t *tmem_slot = misc;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(misc + 1);
    uint32_t *rcnt = misc + 2;                          // readers of a stage, two in turn
    int *n_raw = reinterpret_cast<int *>(misc + 4);    // raw halves issued
    int *n_planes = reinterpret_cast<int *>(misc + 5);  // right-operand stages issued (lincomb)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = su32(sm);
    const int super_k = a.super_k;

    if (tid == 0) {
        for (int s = 0; s < kTcDigStages; ++s) {
            mbar_init(&empty[s], 1);
            mbar_init(&full[s], kTcWarps + (GRAM ? 0 : 1));
        }
        for (int s = 0; s < 4; ++s) mbar_init(&rfull[s], 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&accf[s], 1);
            rcnt[s] = 0;
        }
        mbar_init(fin, 1);
        *abort_flag = 0;
        *n_raw = 0;
        *n_planes = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         su32(tmem_slot)),
                     "r"(kTcTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // bulk copies of raw half h, the k0 + 16 (h % 2) part of the stage at cursor c,
    // into raw buffer h % RH (a linear combination's two halves with the first)
    auto issue_raw = [&](uint32_t h, const TcCursor &c) {
        const uint32_t r = h % RH;
        const uint32_t base = sbase + L::raw_off + r * L::half_bytes;
        const int k0 = c.k0 + 16 * (int)(h & 1);
        if (GRAM) {
            mbar_expect_tx(&rfull[r], (uint32_t)a.mrows * 128u + L::b_box);
            tma_load_2d(base, &mapA, k0, c.w.mt0, &rfull[r]);
            tma_load_2d(base + L::a_box, &mapB, k0, c.w.nt * BN, &rfull[r]);
        } else {
            if (h & 1) return;
            mbar_expect_tx(&rfull[r], 2 * L::a_box);
#pragma unroll
            for (int g = 0; g < kTcM / 16; ++g)
                tma_load_2d(base + g * 4096u, &mapA, c.w.mt0 + 16 * g, k0, &rfull[r]);
        }
        atomicMax(n_raw, (int)h + 1);
    };
    // the MMAs of a stage (buffer s, accumulator set acc, stage st of its chunk, its
    // 16-k steps)
    auto issue_mma = [&](uint32_t s, uint32_t acc, int st, int steps, bool last_of_chunk) {
        const uint32_t abase = sbase + L::dig_off + s * L::stage_bytes;
        const uint32_t bbase = abase + L::a_bytes;
        // left plane i times right planes j = 0 .. 6 - i, into levels l = i + j,
        // in MMAs of at most kLvl levels (N <= 256)
        constexpr int kLvl = 256 / BN < kTcDigits ? 256 / BN : kTcDigits;
#pragma unroll
        for (int ks = 0; ks < kTcStageK / 16; ++ks) {
            if (ks >= steps) break;
#pragma unroll
            for (int i = 0; i < kTcDigits; ++i) {
                const uint64_t ad = smem_desc(abase + i * tc_plane(kTcM) + 2 * ks * tc_lbo(kTcM),
                                              tc_lbo(kTcM), 128);
#pragma unroll
                for (int l0 = i; l0 < kTcDigits; l0 += kLvl) {
                    const int nl = min(kLvl, kTcDigits - l0);
                    const uint64_t bd = smem_desc(bbase + 2 * ks * tc_lbo_b(BN) +
                                                      (uint32_t)((l0 - i) * BN / 8) * 128u,
                                                  tc_lbo_b(BN), 128);
                    // the first product into a level in a drain chunk overwrites it
                    // (level l first meets i = 0)
                    tc_mma(tmem + (acc * kTcDigits + (uint32_t)l0) * BN, ad, bd,
                           tc_idesc(kTcM, nl * BN), (st > 0 || ks > 0 || i > 0) ? 1u : 0u);
                }
            }
        }
        tc_commit(&empty[s]);
        if (last_of_chunk) tc_commit(&accf[acc]);
    };

    if (warp == kTcWarps) {
        // ------------------------------------------------------------ MMA issuer
        uint32_t s = 0, ph = 0;  // ring position and phase of the next stage
        uint32_t acc = 0;        // accumulator set of the chunk
        bool ok = true;
        for (int it = blockIdx.x; it < a.items && ok; it += gridDim.x) {
            const TcItem w = tc_item<GRAM>(a, it);
            for (int sk = w.kb; sk < w.ke && ok; sk += super_k) {
                const int ske = min(w.ke, sk + super_k);
                for (int k0 = sk; k0 < ske && ok; k0 += kTcDrainK) {
                    const int nst = min(kTcDrainStages, (ske - k0 + kTcStageK - 1) / kTcStageK);
                    for (int st = 0; st < nst; ++st) {
                        // every worker finished the stage (and drained the chunk
                        // whose accumulators its first MMAs overwrite)
                        if (!mbar_wait_warp(&full[s], ph, abort_flag, a.error)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const int steps = ske - k0 - st * kTcStageK <= 16 ? 1 : 2;
                        if (tc_elect()) issue_mma(s, acc, st, steps, st == nst - 1);
                        __syncwarp();
                        if (++s == kTcDigStages) s = 0, ph ^= 1;
                    }
                    if (++acc == ACCS) acc = 0;
                }
            }
        }
        // all issued MMAs complete before tensor memory is freed.  A commit tracks
        // the operations of its own thread: the lane that issued them (elect.sync
        // picks the same lane for the same mask every time)
        if (tc_elect()) tc_commit(fin);
        __syncwarp();
        mbar_wait_teardown(fin, 0);
    } else {
        if (tid == 0) {
            TcCursor c;
            cur_init<GRAM>(a, c);
            for (uint32_t h = 0; h < (uint32_t)RH && c.valid; ++h) {
                issue_raw(h, c);
                if (h & 1) cur_next<GRAM>(a, c);
            }
        }

        // Lane = 8 pp + r: row r of a core matrix, k pair pp.  The 4-byte digit
        // stores of a warp fill one 128-byte line, and its reads of a swizzled box
        // (row r's chunk c at c ^ r in a Gram, row pair c of k at c ^ k otherwise)
        // take the fewest bank cycles.
        const int r7 = lane & 7, pp = lane >> 3;
        // drain slice: row q 32 + lane, columns [cp CPW, (cp + 1) CPW)
        constexpr int CPW = BN / 4;
        const int q = warp & 3, cp = warp >> 2;
        const int drow = q * 32 + lane;
        // per column the level sums of the current window, sum over l of
        // L_l 2^(8 (6 - l)), as a 96-bit integer (w0 least significant)
        uint32_t w0[CPW], w1[CPW], w2[CPW];
#pragma unroll
        for (int c = 0; c < CPW; ++c) w0[c] = w1[c] = w2[c] = 0;
        const int amode = a.alpha == 1.0 ? 0 : a.alpha == -1.0 ? 1 : 2;

        // the next chunk to drain: work item, window start, chunk start, its index
        TcItem dw{0, 0, 0, 0};
        int dit = blockIdx.x, dsk = 0, dk0 = 0;
        bool dvalid = dit < a.items;
        uint32_t dn = 0;  // chunks drained
        if (dvalid) {
            dw = tc_item<GRAM>(a, dit);
            dsk = dk0 = dw.kb;
        }
        auto drain = [&]() -> bool {
            const uint32_t acc = dn % ACCS;
            if (!mbar_wait_warp(&accf[acc], (dn / ACCS) & 1, abort_flag, a.error)) return false;
            tc_fence_after();
            // (rows and columns past the operands' are not read)
            const int drows = min(a.mrows, a.M - dw.mt0);
            const bool live = q * 32 < drows && dw.nt * BN + cp * CPW < a.N;
            const uint32_t tb =
                tmem + ((uint32_t)(q * 32) << 16) + acc * kTcDigits * BN + (uint32_t)(cp * CPW);
            // levels 0 and 1, 2 and 3 pair up exactly in 32 bits (|L_0 2^8 + L_1|
            // < 2^30.2, |L_2 2^8 + L_3| < 2^30.9), levels 4 to 6 in 64 with
            // multiply-adds, which stay off the ALU that the digit extraction fills
            auto f2i = [](uint32_t u) { return __float2int_rn(__uint_as_float(u)); };
            if (live) {
#pragma unroll
                for (int j = 0; j < CPW / 4; ++j) {
                    uint32_t u[kTcDigits][4];
#pragma unroll
                    for (int l = 0; l < kTcDigits; ++l) tc_ld4(tb + (uint32_t)(l * BN + 4 * j), u[l]);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int c = 4 * j + e;
                        const int p01 = f2i(u[0][e]) * 256 + f2i(u[1][e]);
                        const int p23 = f2i(u[2][e]) * 256 + f2i(u[3][e]);
                        const long long hi = (long long)p01 * 65536 + p23;  // 2^24
                        const long long lo = (long long)f2i(u[4][e]) * 65536 +
                                             (long long)f2i(u[5][e]) * 256 + f2i(u[6][e]);
                        const uint32_t hl = (uint32_t)hi, hh = (uint32_t)(hi >> 32);
                        tc_acc96(w0[c], w1[c], w2[c], hl << 24, __funnelshift_r(hl, hh, 8),
                                 (uint32_t)((int)hh >> 8));
                        tc_acc96(w0[c], w1[c], w2[c], (uint32_t)lo, (uint32_t)(lo >> 32),
                                 (uint32_t)(lo >> 63));
                    }
                }
            }
            ++dn;
            const int ske = min(dw.ke, dsk + super_k);
            if (dk0 + kTcDrainK >= ske) {
                // the window ends: its sums, w 2^(er + ec - 2106)
                // converted with integer instructions, go into the work item's
                // split-k partial (Gram; a work item of several windows adds
                // them there) or straight into Y (a linear combination)
                const int sidx = (dsk - (GRAM ? 0 : dw.kb)) / super_k;
                const int grow = dw.mt0 + drow;
                const bool row_in = drow < drows;
                const int er = row_in ? __ldg(a.eA + (size_t)sidx * a.M + grow) : 1;
                const bool first = dsk == dw.kb;
                const int z = dit / (a.mtiles * a.ntiles);
#pragma unroll
                for (int c = 0; c < CPW; ++c) {
                    const int col = cp * CPW + c, gcol = dw.nt * BN + col;
                    const int ec = GRAM ? (gcol < a.N ? __ldg(a.eB + (size_t)sidx * a.N + gcol) : 1)
                                        : __ldg(a.eB + ((size_t)dw.nt * a.nsup + sidx) * BN + col);
                    const double val = (er == 0x7FF || ec == 0x7FF)
                                           ? __longlong_as_double(0x7FF8000000000000LL)
                                           : tc_i128_f64((long long)(int)w2[c],
                                                         ((unsigned long long)w1[c] << 32) | w0[c],
                                                         er + ec - 2106);
                    w0[c] = w1[c] = w2[c] = 0;
                    if (GRAM) {
                        // the work item's split-k partial: its first window
                        // writes it, later windows add to it
                        if (row_in && gcol < a.N) {
                            double *dst = a.out + (size_t)z * a.M * a.N + grow + (size_t)gcol * a.M;
                            *dst = first ? val : *dst + val;
                        }
                    } else if (row_in && gcol < a.N) {
                        double *dst = a.out + grow + (size_t)gcol * a.ldo;
                        // alpha = +-1 needs no FP64 multiply (the sign folds
                        // into the beta fma or the store)
                        double y = amode == 0 ? val : amode == 1 ? -val : a.alpha * val;
                        if (a.accumulate) {
                            y += *dst;
                        } else if (a.beta != nullptr) {
                            const double bb = a.beta[a.incb == 0 ? 0 : (size_t)gcol * a.incb];
                            if (bb != 0.0) y = fma(bb, *dst, y);
                        }
                        *dst = y;
                    }
                }
            }
            // the next chunk
            dk0 += kTcDrainK;
            if (dk0 >= ske) {
                dsk += super_k;
                if (dsk >= dw.ke) {
                    dit += gridDim.x;
                    dvalid = dit < a.items;
                    if (dvalid) {
                        dw = tc_item_after<GRAM>(a, dw, dit);
                        dsk = dw.kb;
                    }
                }
                dk0 = dsk;
            }
            return true;
        };

        // ---- production
        TcCursor cons;
        cur_init<GRAM>(a, cons);
        uint32_t t = 0;          // stages produced
        uint32_t chunk = 0;      // chunk of stage t
        uint32_t s = 0, ph = 0;  // ring position and phase of stage t
        // left-operand units of this warp: row group ga, k-groups kg0 .. kg0 + nku - 1;
        // right-operand units (Gram): ub0, ub0 + ubs, .. below nub
        int ga = 0, kg0 = 0, nku = 0, ub0 = 0, ubs = kTcWarps, nub = 0;
        int em_a = 1, em_b0 = 1, em_b1 = 1;  // exponent fields: row; columns lane, lane + 32
        // the field of this lane's row in the tile at mt0 (a linear combination
        // loads the next tile's one tile ahead)
        auto row_field = [&](int mt0, int g, int rows, int sidx) {
            return g * 8 + r7 < rows ? __ldg(a.eA + (size_t)sidx * a.M + mt0 + g * 8 + r7) : 0x7FF;
        };
        int em_next = 0, mt_next = -1;
        bool ok = true;
        while (ok && cons.valid) {
            const int ske = min(cons.w.ke, cons.sk + super_k);
            if (cons.k0 == cons.sk) {
                // a window starts: the units of its tile, and its exponent fields
                const int sidx = (cons.sk - (GRAM ? 0 : cons.w.kb)) / super_k;
                const int rows = min(a.mrows, a.M - cons.w.mt0);
                const int gl = (rows + 7) >> 3;  // row groups: shared by two or four
                                                 // warps where they are few
                const int split = gl > 8 ? 0 : gl > 4 ? 1 : 2;
                ga = warp & (15 >> split);
                nku = gl > ga ? kTcKGroups >> split : 0;
                kg0 = (warp >> (4 - split)) * (kTcKGroups >> split);
                em_a = !GRAM && mt_next == cons.w.mt0 && split == 0
                           ? em_next
                           : row_field(cons.w.mt0, ga, rows, sidx);
                if (!GRAM) {
                    mt_next = tc_item_after<GRAM>(a, cons.w, 0).mt0;
                    em_next = row_field(mt_next, warp, a.M - mt_next, sidx);
                }
                if (GRAM) {
                    const int nc = min(BN, a.N - cons.w.nt * BN);
                    nub = ((nc + 7) >> 3) * kTcKGroups;
                    // to the warps without row groups where they can take them all,
                    // else to all warps in turn
                    const int idle = split == 0 ? kTcWarps - gl : 0;
                    ubs = idle > 0 && nub <= kTcKGroups * idle ? idle : kTcWarps;
                    ub0 = ubs == kTcWarps ? (warp - (int)(t * (uint32_t)nub)) & 15
                                          : (warp >= gl ? warp - gl : nub);
                    const int *e = a.eB + (size_t)sidx * a.N + cons.w.nt * BN;
                    em_b0 = lane < nc ? __ldg(e + lane) : 0x7FF;
                    em_b1 = BN > 32 && lane + 32 < nc ? __ldg(e + lane + 32) : 0x7FF;
                }
            }
            const uint32_t h0 = 2 * t, h1 = h0 + 1;
            if (!mbar_wait_warp(&rfull[h0 % RH], (h0 / RH) & 1, abort_flag, a.error) ||
                (GRAM && !mbar_wait_warp(&rfull[h1 % RH], (h1 / RH) & 1, abort_flag, a.error)))
                break;
            const uint8_t *raw0 = sm + L::raw_off + (h0 % RH) * L::half_bytes;
            const uint8_t *raw1 = sm + L::raw_off + (h1 % RH) * L::half_bytes;
            // a stage's halves are read; the last warp issues the copies of the two
            // that take their buffers
            auto release_raw = [&]() {
                __syncwarp();
                if (lane == 0 && smem_arrive(&rcnt[t & 1]) == kTcWarps - 1) {
                    rcnt[t & 1] = 0;
                    // half h0 + RH belongs to the stage (h0 + RH) / 2
                    TcCursor c2 = cons;
                    uint32_t stage = t;
#pragma unroll 1
                    for (uint32_t h = h0 + RH; h <= h1 + RH; ++h) {
                        for (; stage < h / 2 && c2.valid; ++stage) cur_next<GRAM>(a, c2);
                        if (c2.valid) issue_raw(h, c2);
                    }
                }
                __syncwarp();
            };
            // a linear combination's values are held in registers (its buffers are
            // refilled during the conversion); a Gram's are read unit by unit, as
            // its accumulators and right-operand units need the registers (a spilled
            // one costs an L2 access: shared memory leaves no L1)
            double2 va[GRAM ? 1 : kTcKGroups];
            if (!GRAM) {
#pragma unroll
                for (int u = 0; u < kTcKGroups; ++u) {
                    // box ga / 2: k's 16 rows as 8 chunks of 16 bytes, chunk c at
                    // c ^ (k % 8)
                    const int rr = (ga & 1) * 8 + r7;
                    const int k = (kg0 + min(u, max(nku, 1) - 1)) * 8 + 2 * pp;
                    const uint8_t *box = raw0 + (uint32_t)(ga >> 1) * 4096u + (uint32_t)k * 128u +
                                         (uint32_t)(rr & 1) * 8u;
                    va[u].x = *reinterpret_cast<const double *>(
                        box + ((uint32_t)((rr >> 1) ^ (2 * pp)) << 4));
                    va[u].y = *reinterpret_cast<const double *>(
                        box + 128u + ((uint32_t)((rr >> 1) ^ (2 * pp + 1)) << 4));
                }
                release_raw();
            }
            // the MMAs of stage t - kTcDigStages read this digit buffer
            if (t >= kTcDigStages && !mbar_wait_warp(&empty[s], ph ^ 1, abort_flag, a.error)) break;
            uint8_t *abuf = sm + L::dig_off + s * L::stage_bytes;
            uint8_t *bbuf = abuf + L::a_bytes;
            if (!GRAM && tid == 0) {
                // the right operand's prepared planes of this stage
                mbar_expect_tx(&full[s], L::b_bytes);
                bulk_load(su32(bbuf),
                          a.bplanes + ((size_t)cons.w.nt * a.nstages +
                                       (cons.k0 - cons.w.kb) / kTcStageK) * L::b_bytes,
                          L::b_bytes, &full[s]);
                *n_planes = (int)t + 1;
            }
            if (!GRAM) __syncwarp();
            auto store_a = [&](int kg, const double2 &v) {
                uint32_t d[kTcDigits];
                tc_digit_pair(v.x, v.y, (uint32_t)em_a, d);
                uint8_t *dst = abuf + (uint32_t)kg * tc_lbo(kTcM) + (uint32_t)ga * 128u +
                               (uint32_t)r7 * 16u + (uint32_t)pp * 4u;
#pragma unroll
                for (int i = 0; i < kTcDigits; ++i)
                    *reinterpret_cast<uint32_t *>(dst + (uint32_t)i * tc_plane(kTcM)) = d[i];
            };
            if (!GRAM) {
                // (a stage of at most 16 k is one MMA step: two k-groups; a warp with
                // fewer units repeats its last one instead of branching)
                if (nku > 0 && ske - cons.k0 > 16) {
#pragma unroll
                    for (int u = 0; u < kTcKGroups; ++u) store_a(kg0 + min(u, nku - 1), va[u]);
                } else {
#pragma unroll 1
                    for (int u = 0; u < min(nku, 2 - kg0); ++u)
                        store_a(kg0 + u, u == 0 ? va[0] : va[1]);
                }
            } else {
                constexpr int NU = BN > 32 ? 1 : 2;
#pragma unroll 1
                for (int u = 0; u < nku; u += NU) {
                    double2 v[NU];
#pragma unroll
                    for (int e = 0; e < NU; ++e) {
                        // row's 16 k as 8 chunks of 16 bytes, chunk c at c ^ r7
                        const int kg = kg0 + min(u + e, nku - 1);
                        v[e] = *reinterpret_cast<const double2 *>(
                            ((kg & 2) ? raw1 : raw0) + (uint32_t)(ga * 8 + r7) * 128u +
                            ((uint32_t)((4 * (kg & 1) + pp) ^ r7) << 4));
                    }
#pragma unroll
                    for (int e = 0; e < NU; ++e) store_a(kg0 + min(u + e, nku - 1), v[e]);
                }
            }
            if (GRAM) {
#pragma unroll 1
                for (int b = ub0; b < nub; b += ubs) {
                    const int kg = b & 3, rb = (b >> 2) * 8 + r7;
                    const double2 v = *reinterpret_cast<const double2 *>(
                        ((kg & 2) ? raw1 : raw0) + L::a_box + (uint32_t)rb * 128u +
                        ((uint32_t)((4 * (kg & 1) + pp) ^ r7) << 4));
                    int em = __shfl_sync(0xffffffffu, em_b0, rb & 31);
                    if (BN > 32) {
                        const int e1 = __shfl_sync(0xffffffffu, em_b1, rb & 31);
                        if (rb >= 32) em = e1;
                    }
                    uint32_t d[kTcDigits];
                    tc_digit_pair(v.x, v.y, (uint32_t)em, d);
                    uint8_t *dst = bbuf + (uint32_t)kg * tc_lbo_b(BN) + (uint32_t)rb * 16u +
                                   (uint32_t)pp * 4u;
#pragma unroll
                    for (int i = 0; i < kTcDigits; ++i)
                        *reinterpret_cast<uint32_t *>(dst + (uint32_t)i * BN * 16u) = d[i];
                }
                if (ubs == kTcWarps) ub0 = (ub0 - nub) & 15;
            }
            if (GRAM) release_raw();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            // chunks whose accumulators this stage's chunk overwrites
            while (dvalid && dn + ACCS <= chunk) {
                if (!drain()) {
                    ok = false;
                    break;
                }
            }
            if (!ok) break;
            // arrival (release; the stores and drains above come first)
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if (++s == kTcDigStages) s = 0, ph ^= 1;
            ++t;
            // the next stage starts a chunk at a multiple of the drain length in
            // its window, or with a window
            const int kn = cons.k0 + kTcStageK;
            if (kn >= ske || (kn - cons.sk) % kTcDrainK == 0) ++chunk;
            cur_next<GRAM>(a, cons);
        }
        ok = ok && !cons.valid;
        // the remaining chunks
        while (ok && dvalid)
            if (!drain()) ok = false;
    }
    // teardown: the bulk copies still in flight (after an abort) land before
    // the CTA exits; the MMA warp waited for its MMAs
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        const int nr = *n_raw;
        for (int h = max(nr - RH, 0); h < nr; ++h)
            if (GRAM || (h & 1) == 0) mbar_wait_teardown(&rfull[h % RH], (h / RH) & 1);
        if (!GRAM && *abort_flag) {
            // the right operand's copies arrive on `full`, whose phase an abort
            // leaves incomplete: give them the time any copy takes
            const unsigned long long t0 = tc_global_ns();
            while (*n_planes > 0 && tc_global_ns() - t0 < 1000000ull) {
            }
            __syncwarp();
        }
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTcTmemCols)
                     : "memory");
    }
}

// Exponent fields for the Gram operands: out[s * ncols + c] = the largest
// exponent field (at least 1) of column c of X (n x ncols, leading dimension
// ld, 16-byte aligned columns) over rows [s super, (s + 1) super).  One warp
// per (column, piece of at most kTcExpPiece rows of one window), 16-byte
// loads, merged with atomicMax into `out`, which starts at 0.
constexpr int kTcExpPiece = 4096;
__global__ void __launch_bounds__(256) k_tc_expcols(const double *__restrict__ X, size_t ld,
                                                    int n, int ncols, int super, int nsup,
                                                    int *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int pieces = (super + kTcExpPiece - 1) / kTcExpPiece;  // per window
    const long long units = (long long)nsup * pieces * ncols;
    const long long nw = (long long)gridDim.x * 8;
    for (long long wid = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); wid < units; wid += nw) {
        const int c = (int)(wid % ncols);
        const long long sp = wid / ncols;
        const int s = (int)(sp / pieces), pc = (int)(sp % pieces);
        const int r0 = s * super + pc * kTcExpPiece;
        const int r1 = (int)std::min<long long>(std::min<long long>(n, (long long)(s + 1) * super),
                                                r0 + kTcExpPiece);
        const double *col = X + (size_t)c * ld;
        int em = 1;
#pragma unroll 4
        for (int r = r0 + 2 * lane; r < r1; r += 64) {
            if (r + 1 < r1) {
                const double2 u = __ldg(reinterpret_cast<const double2 *>(col + r));
                em = max(em, max(tc_exp_field(u.x), tc_exp_field(u.y)));
            } else {
                em = max(em, tc_exp_field(__ldg(col + r)));
            }
        }
        em = (int)__reduce_max_sync(0xffffffffu, (unsigned)em);
        if (lane == 0) {
            if (pieces == 1) out[(size_t)s * ncols + c] = em;
            else atomicMax(out + (size_t)s * ncols + c, em);
        }
    }
}
__global__ void __launch_bounds__(256) k_tc_exprows(const double *__restrict__ X, size_t ld,
                                                    int n, int K, int super,
                                                    int *__restrict__ out) {
    const int r = blockIdx.x * 256 + threadIdx.x, s = blockIdx.y;
    if (r >= n) return;
    const int k0 = s * super, k1 = min(K, k0 + super);
    int em = 1;
    int k = k0;
    for (; k + 8 <= k1; k += 8) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = __ldg(X + r + (size_t)(k + q) * ld);
#pragma unroll
        for (int q = 0; q < 8; ++q) em = max(em, tc_exp_field(v[q]));
    }
    for (; k < k1; ++k) em = max(em, tc_exp_field(__ldg(X + r + (size_t)k * ld)));
    out[(size_t)s * n + r] = em;
}

// Right operand of a linear combination (C, K x N, element (k, c) at
// C[k + c ldc]) prepared once per call: block (window, n tile) writes the
// exponent fields of its BN columns and the digit planes of each 32-k digit
// stage of the window in the stage layout of the product kernel.
template <int BN>
__global__ void __launch_bounds__(256) k_tc_bprep(const double *__restrict__ C, size_t ldc, int N,
                                                  int K, int super_k, uint8_t *__restrict__ planes,
                                                  int *__restrict__ exps, int nstages, int nsup) {
    constexpr uint32_t bb = tc_tile_b_bytes(BN);
    __shared__ int em_s[BN];
    const int sidx = blockIdx.x, nt = blockIdx.y;
    const int sk = sidx * super_k, ske = min(K, sk + super_k);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = warp; c < BN; c += 8) {
        const int gc = nt * BN + c;
        int em = 1;
        if (gc < N)
            for (int k = sk + lane; k < ske; k += 32) em = max(em, tc_exp_field(C[k + (size_t)gc * ldc]));
        em = (int)__reduce_max_sync(0xffffffffu, (unsigned)em);
        if (lane == 0) {
            em_s[c] = em;
            exps[((size_t)nt * nsup + sidx) * BN + c] = em;
        }
    }
    __syncthreads();
    for (int k0 = sk; k0 < ske; k0 += kTcStageK) {
        uint8_t *dst = planes + ((size_t)nt * nstages + k0 / kTcStageK) * bb;
        for (int item = threadIdx.x; item < BN * kTcKGroups; item += 256) {
            const int c = item % BN, g = item / BN;
            const int gc = nt * BN + c, k = k0 + g * 8;
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                v[q] = (gc < N && k + q < ske) ? C[k + q + (size_t)gc * ldc] : 0.0;
            uint4 dg[kTcDigits];
            tc_digits8(v, em_s[c], dg);
            uint8_t *base = dst + (uint32_t)g * tc_lbo_b(BN) + (uint32_t)(c >> 3) * 128u +
                            (uint32_t)(c & 7) * 16u;
#pragma unroll
            for (int i = 0; i < kTcDigits; ++i)
                *reinterpret_cast<uint4 *>(base + (uint32_t)i * BN * 16u) = dg[i];
        }
    }
}

// Split-k partial sums in a fixed order: block b sums outputs
// [32 b, 32 b + 32); thread (o, grp) adds partials grp, grp + 8, ... of output
// o, then the 8 groups are added in a fixed tree.
__global__ void __launch_bounds__(256) k_tc_reduce(const double *__restrict__ part, int chunks,
                                                   int m, int w, double *__restrict__ C, int ldc) {
    __shared__ double red[8][33];
    const int total = m * w;
    const int o = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + o;
    double s0 = 0.0, s1 = 0.0;
    if (e < total) {
        int c = grp;
        for (; c + 8 < chunks; c += 16) {
            s0 += part[(size_t)c * total + e];
            s1 += part[(size_t)(c + 8) * total + e];
        }
        if (c < chunks) s0 += part[(size_t)c * total + e];
    }
    red[grp][o] = s0 + s1;
    __syncthreads();
    if (grp == 0 && e < total) {
        const double v = ((red[0][o] + red[1][o]) + (red[2][o] + red[3][o])) +
                         ((red[4][o] + red[5][o]) + (red[6][o] + red[7][o]));
        C[e % m + (size_t)(e / m) * ldc] = v;
    }
}

// Column tile of a right operand of n columns: as many tiles as 48-column ones
// take, of even width (60 columns: two of 32, whose accumulators fit tensor memory
// twice, instead of 48 + 12 in two of 48; 262144 x 40 -> 60 321 us with 16-k stages,
// 357 with two of 48, 249).
int tc_bn(int n) {
    const int tiles = std::max(1, (n + 47) / 48), w = (n + tiles - 1) / tiles;
    return w <= 16 ? 16 : (w <= 32 ? 32 : 48);
}

template <int BN, bool GRAM>
void launch_tc(const CUtensorMap &ma, const CUtensorMap &mb, const TcArgs &a, int grid,
               cudaStream_t st) {
    using L = TcLayout<BN, GRAM>;
    static PerDevice<bool> smem_set;
    smem_set.get([] {
        GCGE_CUDA(cudaFuncSetAttribute(k_tc_digits<BN, GRAM>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)L::alloc_bytes));
        return true;
    });
    k_tc_digits<BN, GRAM><<<grid, kTcThreads, L::alloc_bytes, st>>>(ma, mb, a);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

template <bool GRAM>
void launch_tc_bn(const CUtensorMap &ma, const CUtensorMap &mb, const TcArgs &a, int bn, int grid,
                  cudaStream_t st) {
    switch (bn) {
        case 16: launch_tc<16, GRAM>(ma, mb, a, grid, st); break;
        case 32: launch_tc<32, GRAM>(ma, mb, a, grid, st); break;
        default: launch_tc<48, GRAM>(ma, mb, a, grid, st); break;
    }
}

// Device error word of the product kernels (a wait that ran out), one per
// device; read and cleared by tc_check_error.
int *tc_error_word() {
    static PerDevice<int *> word;
    return word.get([] {
        int *p = nullptr;
        GCGE_CUDA(cudaMalloc((void **)&p, sizeof(int)));
        GCGE_CUDA(cudaMemset(p, 0, sizeof(int)));
        return p;
    });
}

// cuTensorMapEncodeTiled from the driver (the library links the static
// runtime, not the driver library)
PFN_cuTensorMapEncodeTiled_v12000 tc_encode_fn() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                             cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// 2D FP64 tensor map of a column-major block: dim0 (contiguous) x dim1 with
// row pitch ld doubles, box0 x box1 elements (box0 x 8 = the 128-byte swizzle's
// span); false where the layout cannot
// be described (the caller then uses the FP64 kernels).
bool tc_map(CUtensorMap *map, const double *base, int dim0, int dim1, size_t ld, int box0,
            int box1) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tc_encode_fn();
    if (!enc || (reinterpret_cast<uintptr_t>(base) & 15) || (ld * 8) % 16 || dim0 < 1 || dim1 < 1)
        return false;
    const cuuint64_t dims[2] = {(cuuint64_t)dim0, (cuuint64_t)dim1};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 8};
    const cuuint32_t box[2] = {(cuuint32_t)box0, (cuuint32_t)box1};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double *>(base), dims, strides,
               box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t tc_bprep_bytes(int k, int m) {
    const int bn = tc_bn(m);
    const size_t nt = (size_t)(m + bn - 1) / bn;
    const size_t nst = (size_t)(k + kTcStageK - 1) / kTcStageK;
    const size_t nsup = (size_t)(k + kTcSuperLincomb - 1) / kTcSuperLincomb;
    const size_t bb = tc_tile_b_bytes(bn);
    return nt * nst * bb + 256 + nt * nsup * bn * sizeof(int) + 256;
}

}  // namespace

bool tc_digits_available() {
    static PerDevice<int> ok;
    return ok.get([] {
        int major = 0, minor = 0;
        const int dev = current_device();
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
        return (major == 10 && minor == 3 && tc_encode_fn() != nullptr) ? 1 : 0;
    }) != 0;
}

void tc_check_error(cudaStream_t st) {
    int *w = tc_error_word();
    int h = 0;
    GCGE_CUDA(cudaMemcpyAsync(&h, w, sizeof(int), cudaMemcpyDeviceToHost, st));
    GCGE_CUDA(cudaStreamSynchronize(st));
    if (h != 0) {
        GCGE_CUDA(cudaMemsetAsync(w, 0, sizeof(int), st));
        GCGE_CUDA(cudaStreamSynchronize(st));
        throw CudaError{GCGE_ERR_CUDA, "tensor-core digit product: an mbarrier wait timed out"};
    }
}

// C (m x w, ldc) = Q^T P for Q n x m (ldq), P n x w (ldp): split-k partials
// in scratch (scratch_elems doubles), then a fixed-order sum.  Operands that a
// tensor map cannot describe (an odd leading dimension, a base not 16-byte
// aligned) go through the FP64 kernel.
void tc_gram(int n, int m, int w, const double *Q, int ldq, const double *P, int ldp, double *C,
             int ldc, double *scratch, size_t scratch_elems, cudaStream_t st, TcExpCache *cache) {
    if (m <= 0 || w <= 0) return;
    if (n <= 0) {
        GCGE_CUDA(cudaMemset2DAsync(C, sizeof(double) * ldc, 0, sizeof(double) * m, w, st));
        return;
    }
    const int bn = tc_bn(w);
    // row tiles of equal height (180 rows: 96 + 84 instead of 128 + 52, whose
    // CTAs finished at half the time of the others)
    const int mtiles = (m + kTcM - 1) / kTcM;
    const int mrows = ((m + mtiles - 1) / mtiles + 7) / 8 * 8;
    CUtensorMap ma, mb;
    if (!tc_map(&ma, Q, n, m, (size_t)ldq, 16, mrows) ||
        !tc_map(&mb, P, n, w, (size_t)ldp, 16, bn)) {
        gram(n, m, w, Q, ldq, P, ldp, C, ldc, scratch, scratch_elems, st);
        return;
    }
    TcArgs a{};
    a.M = m;
    a.N = w;
    a.K = n;
    a.A = Q;
    a.lda = (size_t)ldq;
    a.mtiles = mtiles;
    a.mrows = mrows;
    a.ntiles = (w + bn - 1) / bn;
    const int mn = a.mtiles * a.ntiles;
    const int sms = device_sms();
    // one wave of one CTA per SM over all work items, fewer and longer k ranges
    // until the partials fit the scratch.  Ranges are whole drain chunks, and
    // whole stages where several tiles share the SMs, whose short ranges a rounding
    // to chunks may double (2000 x 200 x 200: 134 k became 256 and half of the SMs had
    // no item, 52 us, with stages 42; 144-k chunks 44).  With one tile, shorter
    // ranges make a lone short product faster (4160 x 4 x 4 13.1 -> 8.4 us) but
    // take more of the part from other streams: a batch of 256 mixed solves by 8
    // workers 7.46 -> 7.51 s.
    int z = std::max(1, sms / mn);
    const int unit = mn > 1 ? kTcStageK : kTcDrainK;
    long long kc = ((long long)(n + z - 1) / z + unit - 1) / unit * unit;
    GCGE_REQUIRE((size_t)m * w <= scratch_elems, GCGE_ERR_ARG, "tc_gram: scratch too small");
    while ((size_t)((n + kc - 1) / kc) * m * w > scratch_elems) kc *= 2;
    // the exponent window: the whole k range of a work item, or windows of
    // the largest size when the range is longer.  One
    // exponent per column over K rows bounds the error of an entry by
    // 2^-54 sqrt(K) |x| |y|, below the FP64 dot product's K 2^-53 |x| |y|.
    if (kc > kTcSuperGramMax) kc = (kc + kTcSuperGramMax - 1) / kTcSuperGramMax * kTcSuperGramMax;
    const int super_k = (int)std::min<long long>(kc, kTcSuperGramMax);
    z = (int)((n + kc - 1) / kc);
    a.super_k = super_k;
    const int nsup = (n + super_k - 1) / super_k;
    const long long pieces = (super_k + kTcExpPiece - 1) / kTcExpPiece;
    auto expcols = [&](const double *X, int ld, int cols, int *out) {
        if (pieces > 1) GCGE_CUDA(cudaMemsetAsync(out, 0, sizeof(int) * (size_t)nsup * cols, st));
        const int gx = (int)std::min<long long>(8 * sms, (nsup * pieces * cols + 7) / 8);
        k_tc_expcols<<<gx, 256, 0, st>>>(X, (size_t)ld, n, cols, super_k, nsup, out);
        GCGE_CHECK_LAUNCH();
        count_launch();
    };
    DevBuf<int> &eb = slot_stage().tc_exps;
    int *eA, *eB;
    if (cache) {
        // Q's fields from the cache (computed there on first use)
        if (!cache->matches(Q, (size_t)ldq, n, m, super_k, 0)) {
            cache->e.alloc((size_t)nsup * m);
            expcols(Q, ldq, m, cache->e.p);
            cache->set(Q, (size_t)ldq, n, m, super_k, 0);
        }
        eA = cache->e.p;
        eb.alloc((size_t)nsup * w);
        eB = eb.p;
    } else {
        eb.alloc((size_t)nsup * (m + w));
        eA = eb.p;
        eB = eb.p + (size_t)nsup * m;
        expcols(Q, ldq, m, eA);
    }
    expcols(P, ldp, w, eB);
    a.eA = eA;
    a.eB = eB;
    a.kchunk = (int)kc;
    a.items = z * mn;
    a.out = scratch;
    a.error = tc_error_word();
    launch_tc_bn<true>(ma, mb, a, bn, std::min(a.items, sms), st);
    const int tot = m * w;
    k_tc_reduce<<<(tot + 31) / 32, 256, 0, st>>>(scratch, z, m, w, C, ldc);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

size_t tc_lincomb_scratch_bytes(int k, int m) {
    return tc_bprep_bytes(std::min(k, kTcSuperLincomb), m);
}

// Y (n x m, ldy) = alpha X C + Y diag(beta) for X n x k (ldx), C k x m (ldc);
// beta == nullptr overwrites Y; incb == 0 broadcasts beta[0].  Contractions
// longer than one window (432) run as several launches, each later one
// adding its block's product to Y.
void tc_lincomb(int n, int k, int m, const double *X, int ldx, const double *C, int ldc, double *Y,
                int ldy, const double *beta_dev, int incb, cudaStream_t st, double alpha,
                void *scratch, size_t scratch_bytes, TcExpCache *cache) {
    if (n <= 0 || m <= 0) return;
    const int bn = tc_bn(m);
    CUtensorMap ma;
    if (!tc_map(&ma, X, n, std::min(k, kTcSuperLincomb), (size_t)ldx, 16, kTcStageK)) {
        lincomb(n, k, m, X, ldx, C, ldc, Y, ldy, beta_dev, incb, st, alpha);
        return;
    }
    GCGE_REQUIRE(scratch && scratch_bytes >= tc_lincomb_scratch_bytes(k, m), GCGE_ERR_ARG,
                 "tc_lincomb: scratch too small");
    for (int k0 = 0; k0 < k; k0 += kTcSuperLincomb) {
        const int kb = std::min(kTcSuperLincomb, k - k0);
        const double *Xb = X + (size_t)k0 * ldx;
        // (the first block's map was made above; Xb keeps its 16-byte alignment)
        if (k0 > 0 && !tc_map(&ma, Xb, n, kb, (size_t)ldx, 16, kTcStageK))
            throw CudaError{GCGE_ERR_ARG, "tc_lincomb: operand layout"};
        TcArgs a{};
        a.M = n;
        a.N = m;
        a.K = kb;
        a.A = Xb;
        a.lda = (size_t)ldx;
        a.super_k = kTcSuperLincomb;
        a.mtiles = (n + kTcM - 1) / kTcM;
        a.mrows = kTcM;
        a.ntiles = (m + bn - 1) / bn;
        a.items = a.mtiles * a.ntiles;
        a.out = Y;
        a.ldo = (size_t)ldy;
        a.beta = beta_dev;
        a.incb = incb;
        a.alpha = alpha;
        a.accumulate = k0 > 0 ? 1 : 0;
        a.nstages = (kb + kTcStageK - 1) / kTcStageK;
        a.nsup = 1;
        a.error = tc_error_word();
        uint8_t *planes = static_cast<uint8_t *>(scratch);
        const size_t pbytes = (size_t)a.ntiles * a.nstages * tc_tile_b_bytes(bn);
        int *bexps = reinterpret_cast<int *>(
            (reinterpret_cast<uintptr_t>(planes + pbytes) + 255) & ~(uintptr_t)255);
        const dim3 pg(1, a.ntiles);
        const double *Cb = C + k0;
        switch (bn) {
            case 16: k_tc_bprep<16><<<pg, 256, 0, st>>>(Cb, (size_t)ldc, m, kb, kTcSuperLincomb, planes, bexps, a.nstages, 1); break;
            case 32: k_tc_bprep<32><<<pg, 256, 0, st>>>(Cb, (size_t)ldc, m, kb, kTcSuperLincomb, planes, bexps, a.nstages, 1); break;
            default: k_tc_bprep<48><<<pg, 256, 0, st>>>(Cb, (size_t)ldc, m, kb, kTcSuperLincomb, planes, bexps, a.nstages, 1); break;
        }
        // exponent fields of the rows of X over the block's columns (kept in
        // the cache when the whole contraction is one block)
        const bool cached = cache != nullptr && k <= kTcSuperLincomb;
        DevBuf<int> &eb = cached ? cache->e : slot_stage().tc_exps;
        count_launch();
        if (!cached || !cache->matches(Xb, (size_t)ldx, n, kb, kTcSuperLincomb, 1)) {
            eb.alloc((size_t)n);
            k_tc_exprows<<<dim3((n + 255) / 256, 1), 256, 0, st>>>(Xb, (size_t)ldx, n, kb,
                                                                 kTcSuperLincomb, eb.p);
            GCGE_CHECK_LAUNCH();
            count_launch();
            if (cached) cache->set(Xb, (size_t)ldx, n, kb, kTcSuperLincomb, 1);
        }
        a.bplanes = planes;
        a.eA = eb.p;
        a.eB = bexps;
        launch_tc_bn<false>(ma, ma, a, bn, std::min(a.items, device_sms()), st);
    }
}

}  // namespace gcge
