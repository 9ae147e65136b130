// Block conjugate gradient on (A + sigma B) x = b for all columns of a block
// at once (reference BlockPCG, src/ops_lin_sol.c:140-437).
//
// The whole solve is ONE persistent kernel launch (cooperative grid, or one
// thread-block cluster for small operators, below).  Each block
// owns a contiguous range of SELL slices (balanced by stored entries) and the
// rows they cover; the iteration runs in three phases separated by grid-wide
// barriers:
//   1. p = r + beta p                      (own rows; p = r on the first step)
//   2. w = S p, partial sums of p^T w      (warp per slice, gathers p rows)
//      -> every block sums the blocks' partials: alpha = rho / p^T w
//   3. x += alpha p, r -= alpha w, partial sums of r^T r
//      -> residual norms, convergence test, beta, count
// so nothing returns to the host between iterations.  The reference keeps a
// compacted list of unconverged columns and runs one SpMM per contiguous run
// of them; here a per-column `active` flag plays that role: inactive columns
// keep x and r (alpha = 0), drop out of the sums, and a 16-byte group of
// columns that is wholly inactive is neither gathered nor updated.
//
// Every block takes the cross-block sums for itself, all in the same fixed order,
// so results are deterministic for a given grid.  (With two blocks an SM, the
// last of them to arrive summing for all and the scalars in global memory, the
// barriers took 20 us of a step of 92 at 64^3 with 27 points and 20 columns.)  The shifted operator is one SELL matrix
// S = A + sigma B on the union pattern of A and B (the reference's in-place
// MatAxpby branch, src/ops_eig_sol_gcg.c:600-608), so each iteration streams
// one matrix.  Vectors are slice-blocked n x kp blocks (kp = k padded to 16
// bytes, G = kp / (16 / sizeof T) 16-byte column groups; for every 32-row
// slice, group u of its 32 rows is one contiguous 512-byte run): a lane owns
// a row and gathers a neighbour row as G 16-byte loads, and for a stencil the
// 32 lanes of a warp read one or two contiguous runs per load instead of 32
// scattered rows.  T = double (FP64 GCG) or float (mixed precision: FP32
// values and FP32 accumulation within a block; cross-block sums in double).
//
// Every grid-barrier wait is bounded (time and poll count); a wait that runs out
// sets an error flag that makes all blocks return, and the host reports it.  The
// cluster form below waits at the hardware's cluster barrier, which has no bound:
// the cluster's blocks are scheduled together and wait for nobody else.
//
// Small operators, whose steps are bound by the barriers and by the latency of
// each phase instead, run k_pcg_small (below).
//
// (Included by pcg.cu and pcg_f64.cu, which instantiate it for FP32 and FP64:
// the widths take a minute to compile.)
#pragma once
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "pcg.cuh"

namespace gcge {

namespace {

constexpr unsigned long long kBarrierTimeoutNs = 4000000000ull;  // 4 s
constexpr long long kBarrierMaxPolls = 1LL << 27;

// 16-byte packs of a slice-blocked block
template <typename T>
struct Pk;
template <>
struct Pk<float> {
    static constexpr int L = 4;
    float v[4];
    __device__ __forceinline__ static Pk ld(const float *p) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        return Pk{{t.x, t.y, t.z, t.w}};
    }
    __device__ __forceinline__ void st(float *p) const {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <>
struct Pk<double> {
    static constexpr int L = 2;
    double v[2];
    __device__ __forceinline__ static Pk ld(const double *p) {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        return Pk{{t.x, t.y}};
    }
    __device__ __forceinline__ void st(double *p) const {
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    }
};

// Element offset of row i, 16-byte group u in a slice-blocked block of width KP.
template <typename T, int KP>
__device__ __forceinline__ size_t boff(int i, int u) {
    constexpr int L = Pk<T>::L, G = KP / L;
    return ((size_t)(i >> 5) * G + u) * (32 * L) + (size_t)(i & 31) * L;
}

// acc += sum over the lane's row of a slice of val[e] * X(col[e], :), e =
// e0 + 32 i, i < width: the column indices and values of the next kPrefetch
// entries are in flight while the current entry's 16-byte groups are gathered,
// so the gathers do not wait on the matrix stream.  Groups with ga[u] false
// are skipped.
constexpr int kPrefetch = 2;
template <typename T, int KP>
__device__ __forceinline__ void gather_row(const int *__restrict__ col, const T *__restrict__ val,
                                           long long e0, int width, const T *X,
                                           const bool (&ga)[KP / Pk<T>::L], T (&acc)[KP]) {
    constexpr int L = Pk<T>::L, G = KP / L;
    int jq[kPrefetch];
    T vq[kPrefetch];
#pragma unroll
    for (int d = 0; d < kPrefetch; ++d) {
        const bool in = d < width;
        jq[d] = in ? __ldg(col + e0 + 32LL * d) : 0;
        vq[d] = in ? __ldg(val + e0 + 32LL * d) : T(0);
    }
#pragma unroll 1
    for (int e = 0; e < width; ++e) {
        const int j = jq[0];
        const T v = vq[0];
#pragma unroll
        for (int d = 0; d + 1 < kPrefetch; ++d) {
            jq[d] = jq[d + 1];
            vq[d] = vq[d + 1];
        }
        const int en = e + kPrefetch;
        jq[kPrefetch - 1] = en < width ? __ldg(col + e0 + 32LL * en) : 0;
        vq[kPrefetch - 1] = en < width ? __ldg(val + e0 + 32LL * en) : T(0);
#pragma unroll
        for (int u = 0; u < G; ++u) {
            if (!ga[u]) continue;
            const Pk<T> x = Pk<T>::ld(X + boff<T, KP>(j, u));
#pragma unroll
            for (int q = 0; q < L; ++q) acc[u * L + q] = fma(v, x.v[q], acc[u * L + q]);
        }
    }
}

// The same sum for the NU column groups [U0, U0 + NU) only (all of them,
// active or not), two matrix entries at a time (both entries' loads in
// flight before their FMAs): the SpMM phase of wide blocks gathers a row in
// two such halves, so that the accumulators of one half leave registers for
// the second entry's loads (4.87 -> 4.75 s of inner solve per 128^3 solve;
// four entries at a time: 4.81 s).
template <typename T, int KP, int U0, int NU, int NE>
__device__ __forceinline__ void gather_entries(const int *__restrict__ col,
                                               const T *__restrict__ val, long long e0, int e,
                                               const T *X, T (&acc)[NU * Pk<T>::L]) {
    constexpr int L = Pk<T>::L;
    int j[NE];
    T v[NE];
#pragma unroll
    for (int d = 0; d < NE; ++d) {
        j[d] = __ldg(col + e0 + 32LL * (e + d));
        v[d] = __ldg(val + e0 + 32LL * (e + d));
    }
    Pk<T> x[NE][NU];
#pragma unroll
    for (int d = 0; d < NE; ++d)
#pragma unroll
        for (int u = 0; u < NU; ++u) x[d][u] = Pk<T>::ld(X + boff<T, KP>(j[d], U0 + u));
#pragma unroll
    for (int d = 0; d < NE; ++d)
#pragma unroll
        for (int u = 0; u < NU; ++u)
#pragma unroll
            for (int q = 0; q < L; ++q) acc[u * L + q] = fma(v[d], x[d][u].v[q], acc[u * L + q]);
}
template <typename T, int KP, int U0, int NU>
__device__ __forceinline__ void gather_row_part(const int *__restrict__ col,
                                                const T *__restrict__ val, long long e0,
                                                int width, const T *X, T (&acc)[NU * Pk<T>::L]) {
    int e = 0;
#pragma unroll 1
    for (; e + 1 < width; e += 2) gather_entries<T, KP, U0, NU, 2>(col, val, e0, e, X, acc);
    if (e < width) gather_entries<T, KP, U0, NU, 1>(col, val, e0, e, X, acc);
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier number `epoch` (1, 2, ...): every block waits for the
// arrivals of all.  Returns false when the wait ran out (or another block's
// did); the caller then returns.
__device__ __forceinline__ bool grid_arrive_wait(PcgSync *gs, int *error,
                                                 unsigned long long timeout_ns,
                                                 long long max_polls, unsigned long long epoch) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_ok = 1;
        __threadfence();
        const unsigned long long all = epoch * gridDim.x;
        if (atomicAdd(&gs->arrive, 1ull) + 1ull < all) {
            const unsigned long long t0 = global_ns();
            for (long long poll = 0; ld_acquire(&gs->arrive) < all; ++poll) {
                if ((poll & 31) == 31 &&
                    (*(volatile int *)error != 0 || poll > max_polls ||
                     global_ns() - t0 > timeout_ns)) {
                    atomicExch(error, 1);
                    s_ok = 0;
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
}

template <typename T>
struct PcgArgs {
    const long long *sp;
    const int *col;
    const T *val;
    int n, nslices;
    long long stored;  // entries of the SELL arrays, padding included
    const T *B;
    T *X, *R, *P, *W;
    int k, max_iter, rel_tol, x_zero;
    double rate, tol;
    double matrix_bytes;  // nnz (v + 4) + 4 (n + 1) of S
    PcgScalars *sc;
    PcgSync *sync;
    PcgStats *stats;
    double *part;  // two sets (by barrier parity) of 2 x gridDim.x x kp
    // bound of every grid-barrier wait (device clock and poll count)
    unsigned long long timeout_ns;
    long long max_polls;
    // failure-detection test only: the grid's last block returns before its
    // first barrier, so the others' waits run out (never set otherwise)
    int withhold_last;
};

// What a launch adds to PcgStats, kept in shared memory by one thread until the
// launch ends.
template <typename T>
struct PcgTally {
    unsigned long long t0, ns;
    long long groups;  // active 16-byte column groups, summed over the steps
    int steps;
    __device__ void clear() { ns = 0, groups = 0, steps = 0; }
    __device__ void begin() { t0 = global_ns(); }
    __device__ void end(int active_groups) {
        ns += global_ns() - t0;
        groups += active_groups;
        ++steps;
    }
    __device__ void write(const PcgArgs<T> &a, int kp) const {
        const double vec = (double)a.n * 16.0 * groups, start = 4.0 * a.n * kp * sizeof(T);
        a.stats->spmm_ns += ns;
        // SpMM: the matrix once, p read once, w written once
        a.stats->spmm_bytes += steps * a.matrix_bytes + 2.0 * vec;
        // step: p update (r, p read; p written), SpMM (p gathered and re-read, w
        // written), x and r update (x, p, r, w read; x, r written)
        a.stats->kernel_bytes +=
            (a.x_zero ? 0.0 : a.matrix_bytes) + start + steps * a.matrix_bytes + 12.0 * vec;
    }
};

// Compiler-only ordering point between the 16-byte groups of a row in the
// streaming phases: keeps one group's loads in flight per thread instead of
// all of them, which bounds the registers (warps supply the parallelism).
__device__ __forceinline__ void group_fence() { asm volatile("" ::: "memory"); }

__host__ __device__ constexpr int pow2ceil(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// Warp sums of N per-lane column values (N a power of two <= 32): returns, in
// lane l, the sum over the 32 lanes of column l % N.  The first log2(N) steps
// exchange halves of the values between lanes (a transposing butterfly), the
// others add single values: N - 1 + log2(32 / N) additions.  FP64 additions
// occupy a scheduler for 64 clocks each.
template <typename T, int N>
__device__ __forceinline__ T warp_cols_reduce(T (&v)[N], int lane) {
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const T send = up ? v[i] : v[i + h];
            const T keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    T s = v[0];
#pragma unroll
    for (int o = 16; o >= N; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Adds the warp's column sums of acc[0..KP) to wrow[0..KP) (this warp's row of
// shared accumulators; lane c owns column c).
template <typename T, int KP>
__device__ __forceinline__ void warp_cols_add(const T (&acc)[KP], double *wrow, int lane) {
    constexpr int K1 = KP < 32 ? KP : 32;
    constexpr int N1 = pow2ceil(K1);
    T v[N1];
#pragma unroll
    for (int i = 0; i < N1; ++i) v[i] = i < K1 ? acc[i] : T(0);
    const T s = warp_cols_reduce<T, N1>(v, lane);
    if (lane < K1) wrow[lane] += (double)s;
    if constexpr (KP > 32) {
        constexpr int K2 = KP - 32;
        constexpr int N2 = pow2ceil(K2);
        T u[N2];
#pragma unroll
        for (int i = 0; i < N2; ++i) u[i] = i < K2 ? acc[32 + i] : T(0);
        const T s2 = warp_cols_reduce<T, N2>(u, lane);
        if (lane < K2) wrow[32 + lane] += (double)s2;
    }
}

// Column sums over `count` values get(b, c): Q lanes of a warp a column, each every
// Q-th value, then a tree over the lanes; use(c, sum, q) on all of them.  (An
// FP64 addition occupies a scheduler for 64 clocks whatever the lanes at work:
// a column's chain is kept short and few warps take part.)
template <typename Get, typename Use>
__device__ __forceinline__ void lane_cols_sum(int kp, int count, Get get, Use use) {
    const int tid = threadIdx.x, Q = kp <= 16 ? 8 : 4;
    if (tid >= ((kp * Q + 31) & ~31)) return;
    const int c = tid / Q, q = tid % Q;
    double t = 0.0;
    if (c < kp && q < count) {
        t = get(q, c);
        for (int b = q + Q; b < count; b += Q) t += get(b, c);
    }
    for (int o = Q / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (c < kp) use(c, t, q);
}

// Sums of the columns of the nb block partials part[b * kp + c], taken by every
// block for itself; use(c, sum) on one lane each, and the caller synchronises the
// block.  `stripes` threads a column first add a fixed share of the blocks.
template <int NT, typename Use>
__device__ __forceinline__ void grid_cols_sum(const double *part, int nb, int kp, double *stripe,
                                              Use use) {
    const int stripes = min(min(NT / kp, 32), nb);
    const int c = threadIdx.x % kp, st = threadIdx.x / kp;
    if (st < stripes) {  // L2 loads: other blocks wrote them
        double t0 = __ldcg(part + (size_t)st * kp + c);
        double t1 = 0.0;
        int b = st + stripes;
        if (b < nb) t1 = __ldcg(part + (size_t)b * kp + c);
        for (b += stripes; b + stripes < nb; b += 2 * stripes) {
            const double v0 = __ldcg(part + (size_t)b * kp + c);
            const double v1 = __ldcg(part + (size_t)(b + stripes) * kp + c);
            t0 += v0;
            t1 += v1;
        }
        if (b < nb) t0 += __ldcg(part + (size_t)b * kp + c);
        stripe[threadIdx.x] = t0 + t1;
    }
    __syncthreads();
    lane_cols_sum(
        kp, stripes, [&](int i, int col) { return stripe[i * kp + col]; },
        [&](int col, double t, int q) {
            if (q == 0) use(col, t);
        });
}

// a / b for a coefficient that is used in T.  For FP32 a quotient that rounds to the
// same FP32 value: the divisor's reciprocal in FP32 and one Newton step in FP64,
// y + y (1 - b y), whose relative error is at most (2^-23)^2 and a rounding, below
// 130 units in the last place; three dependent FP64 operations instead of a
// division's chain.  The division decides where that is too close to the middle of
// two FP32 values (bits 28..0 at 2^28) or outside the normal FP32 range.  The tests
// are on the bits: an FP64 comparison occupies a scheduler for 64 clocks (four of
// them took 6.4 us of 138 in 30 steps at n = 4160, k = 4).
template <typename T>
__device__ __forceinline__ double scalar_quotient(double a, double b) {
    if constexpr (sizeof(T) == 4) {
        auto exponent = [](double v) { return ((unsigned)__double2hiint(v) >> 20) & 0x7ffu; };
        if (exponent(b) - (1023u - 99u) < 199u) {  // 2^-99 <= |b| < 2^100
            const double y = (double)(1.0f / (float)b);
            const double q = a * fma(y, fma(-b, y, 1.0), y);
            const int past = (__double2loint(q) & 0x1fffffff) - 0x10000000;
            // 2^-125 <= |q| < 2^127, and past the middle by twice the error
            if (exponent(q) - (1023u - 125u) < 252u && abs(past) > 256) return q;
        }
    }
    return a / b;
}

// The r^T r at and below which a column leaves, !(|r| > u && |r| > v) on squares
// (src/ops_lin_sol.c:383-394): negative bounds never stop a column, one that is
// not a number does at once.
__device__ __forceinline__ double stop_square(double u, double v) {
    if (u != u || v != v) return u + v;
    const double m = fmax(u, v);
    return m < 0.0 ? -1.0 : m * m;
}

// Wide blocks (at least 8 column groups, an even number) gather the SpMM
// phase in two halves of the column groups.
template <typename T, int KP>
constexpr bool kSplitGather = (KP / Pk<T>::L) >= 8 && (KP / Pk<T>::L) % 2 == 0;

// Block shape by row width, one block per SM: 1024 threads (<= 64 registers) for
// rows up to 80 bytes and for FP32 rows of 40 columns (whose phases run in two
// column parts: twice the warps hiding gather latency of 512 threads), 512
// threads up to 160 bytes, and 256 threads for wider FP64 rows.
template <typename T, int KP>
__host__ __device__ constexpr int pcg_threads() {
    return sizeof(T) * KP <= 80 || (sizeof(T) == 4 && KP == 40) ? 1024
           : sizeof(T) * KP <= 160                              ? 512
                                                                : 256;
}

template <typename T, int KP>
__global__ void __launch_bounds__(pcg_threads<T, KP>(), 1)
k_block_pcg(PcgArgs<T> a) {
    constexpr int kPcgThreads = pcg_threads<T, KP>();
    constexpr int L = Pk<T>::L;
    constexpr int G = KP / L;  // 16-byte groups per row
    constexpr int nwarps = kPcgThreads / 32;
    // column-group parts of the setup, SpMM and update phases
    constexpr int NP = kSplitGather<T, KP> ? 2 : 1;
    constexpr int GP = G / NP, KPP = KP / NP;
    auto for_parts = [](auto &&f) {
        f(std::integral_constant<int, 0>{});
        if constexpr (NP == 2) f(std::integral_constant<int, 1>{});
    };
    __shared__ double wred[nwarps][KP];  // per-warp column sums of one phase
    __shared__ double stripe[kPcgThreads];
    __shared__ double sums[2][KP];
    __shared__ double stop[KP];  // r^T r at which a column leaves
    __shared__ PcgScalars s_sc;  // every block's own, all the same
    __shared__ T s_coef[KP];
    __shared__ int s_act[KP];
    __shared__ int s_gact[G];
    __shared__ int s_nactive;
    __shared__ long long s_range[2];

    PcgScalars *sc = &s_sc;
    PcgSync *gs = a.sync;
    int *error = &a.sync->error;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = a.k, n = a.n;
    if (a.withhold_last && gridDim.x > 1 && blockIdx.x == gridDim.x - 1) return;

    const bool stats_thread = blockIdx.x == 0 && tid == kPcgThreads - 1;
    __shared__ PcgTally<T> tally;
    if (stats_thread) tally.clear();
    const int nb = gridDim.x;
    unsigned long long epoch = 0;
    // Two sets of partials alternate by the barrier's parity: blocks read them
    // after a barrier while faster ones already write the next phase's.
    auto part_of = [&](unsigned long long e, int which) {
        return a.part + ((size_t)(e & 1) * 2 + which) * nb * KP;
    };
    // per-warp accumulators: clear, and this block's sums for the next barrier
    auto wred_zero = [&]() {
        for (int i = tid; i < nwarps * KP; i += kPcgThreads) (&wred[0][0])[i] = 0.0;
        __syncthreads();
    };
    auto publish = [&](int which) {
        __syncthreads();
        lane_cols_sum(
            KP, nwarps, [&](int w, int c) { return wred[w][c]; },
            [&](int c, double t, int q) {
                if (q == 0) part_of(epoch + 1, which)[(size_t)blockIdx.x * KP + c] = t;
            });
        __syncthreads();
    };
    auto total = [&](int which, auto use) {
        grid_cols_sum<kPcgThreads>(part_of(epoch, which), nb, KP, stripe, use);
    };
    auto barrier = [&]() {
        return grid_arrive_wait(gs, error, a.timeout_ns, a.max_polls, ++epoch);
    };

    // slice range of this block, balanced by stored entries
    if (tid < 2) {
        const long long total = a.sp[a.nslices];
        const long long target = total * (long long)(blockIdx.x + tid) / gridDim.x;
        int lo = 0, hi = a.nslices;  // first slice s with sp[s] >= target
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (a.sp[mid] < target) lo = mid + 1;
            else hi = mid;
        }
        s_range[tid] = (blockIdx.x + tid == gridDim.x) ? a.nslices : lo;
    }
    __syncthreads();
    const int s0 = (int)s_range[0], s1 = (int)s_range[1];
    const int r0 = min(n, 32 * s0), r1 = min(n, 32 * s1);

    auto finish = [&](bool ok) {
        __syncthreads();
        if (blockIdx.x == 0) {  // the host reads the first block's scalars
            if (tid < k) sc->last_res[tid] = sqrt(sc->rho2[tid]);
            __syncthreads();
            const int *src = reinterpret_cast<const int *>(sc);
            int *dst = reinterpret_cast<int *>(a.sc);
            for (int i = tid; i < (int)(sizeof(PcgScalars) / sizeof(int)); i += kPcgThreads)
                dst[i] = src[i];
            if (tid == 0) {
                if (!ok || *(volatile int *)error) a.stats->error = 1;
                a.stats->launches += 1;
                a.stats->iters += (unsigned long long)sc->niter;
            }
            if (stats_thread) tally.write(a, KP);
        }
    };

    // ---------------- r = b - S x (or r = b for x = 0), p = 0, norms
    // (wide blocks work on their column groups in parts, which bounds the
    // accumulator registers of every phase)
    wred_zero();
    if (a.x_zero) {
        for_parts([&](auto part) {
            constexpr int U0 = decltype(part)::value * GP;
            T racc[KPP];
#pragma unroll
            for (int c = 0; c < KPP; ++c) racc[c] = T(0);
            for (int row = r0 + tid; row < r1; row += kPcgThreads) {
#pragma unroll
                for (int uu = 0; uu < GP; ++uu) {
                    const int u = U0 + uu;
                    const Pk<T> b = Pk<T>::ld(a.B + boff<T, KP>(row, u));
                    Pk<T> z;
#pragma unroll
                    for (int q = 0; q < L; ++q) {
                        z.v[q] = T(0);
                        racc[uu * L + q] = fma(b.v[q], b.v[q], racc[uu * L + q]);
                    }
                    b.st(a.R + boff<T, KP>(row, u));
                    z.st(a.X + boff<T, KP>(row, u));
                    z.st(a.P + boff<T, KP>(row, u));
                    group_fence();
                }
            }
            warp_cols_add<T, KPP>(racc, wred[warp] + U0 * L, lane);
        });
    } else {
        for (int s = s0 + warp; s < s1; s += nwarps) {
            const long long beg = a.sp[s], end = a.sp[s + 1];
            const int row = s * 32 + lane;
            for_parts([&](auto part) {
                constexpr int U0 = decltype(part)::value * GP;
                T acc[KPP];
#pragma unroll
                for (int c = 0; c < KPP; ++c) acc[c] = T(0);
                gather_row_part<T, KP, U0, GP>(a.col, a.val, beg + lane, (int)((end - beg) >> 5),
                                               a.X, acc);
                if (row < n) {
#pragma unroll
                    for (int uu = 0; uu < GP; ++uu) {
                        const int u = U0 + uu;
                        const Pk<T> b = Pk<T>::ld(a.B + boff<T, KP>(row, u));
                        Pk<T> r, z;
#pragma unroll
                        for (int q = 0; q < L; ++q) {
                            r.v[q] = b.v[q] - acc[uu * L + q];
                            z.v[q] = T(0);
                            acc[uu * L + q] = r.v[q] * r.v[q];
                        }
                        r.st(a.R + boff<T, KP>(row, u));
                        z.st(a.P + boff<T, KP>(row, u));
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < KPP; ++c) acc[c] = T(0);
                }
                warp_cols_add<T, KPP>(acc, wred[warp] + U0 * L, lane);
            });
        }
    }
    publish(0);
    if (a.rel_tol) {
        wred_zero();
        for_parts([&](auto part) {
            constexpr int U0 = decltype(part)::value * GP;
            T bacc[KPP];
#pragma unroll
            for (int c = 0; c < KPP; ++c) bacc[c] = T(0);
            for (int row = r0 + tid; row < r1; row += kPcgThreads) {
#pragma unroll
                for (int uu = 0; uu < GP; ++uu) {
                    const Pk<T> b = Pk<T>::ld(a.B + boff<T, KP>(row, U0 + uu));
#pragma unroll
                    for (int q = 0; q < L; ++q)
                        bacc[uu * L + q] = fma(b.v[q], b.v[q], bacc[uu * L + q]);
                    group_fence();
                }
            }
            warp_cols_add<T, KPP>(bacc, wred[warp] + U0 * L, lane);
        });
        publish(1);
    }
    if (!barrier()) {
        if (tid == 0) sc->niter = 0;
        finish(false);
        return;
    }
    // initial residual norms (src/ops_lin_sol.c:171-233)
    total(0, [&](int c, double v) { sums[0][c] = v; });
    if (a.rel_tol) {
        __syncthreads();
        total(1, [&](int c, double v) { sums[1][c] = v; });
    }
    __syncthreads();
    if (tid < kPcgMaxCols) {
        const int c = tid;
        int on = 0;
        if (c < k) {
            const double nrm = a.rel_tol ? sqrt(sums[1][c]) : 1.0;
            const double rr = sums[0][c], res = sqrt(rr);
            sc->norm_b[c] = nrm;
            sc->rho2[c] = rr;
            sc->init_res[c] = res;
            sc->last_res[c] = res;
            sc->alpha[c] = sc->beta[c] = 0.0;
            on = res > a.tol * nrm ? 1 : 0;
            stop[c] = stop_square(a.rate * res, a.tol * nrm);
        }
        sc->active[c] = on;
        sc->left_at[c] = 0;
        if (c < KP) {
            s_act[c] = on;
            s_coef[c] = T(0);  // beta of the first step
        }
    }
    __syncthreads();
    if (tid == 0) {
        int cnt = 0;
        for (int c = 0; c < k; ++c) cnt += s_act[c];
        s_nactive = sc->nactive = cnt;
        sc->niter = 0;
    }
    __syncthreads();

    for (int it = 0; it < a.max_iter && s_nactive > 0; ++it) {
        // ---------------- phase 1: p = r + beta p
        if (tid < G) {
            int any = 0;
            for (int q = 0; q < L; ++q) any |= s_act[tid * L + q];
            s_gact[tid] = any;
        }
        __syncthreads();
        const bool first = it == 0;
        for (int row = r0 + tid; row < r1; row += kPcgThreads) {
#pragma unroll
            for (int u = 0; u < G; ++u) {
                if (!s_gact[u]) continue;
                const Pk<T> r = Pk<T>::ld(a.R + boff<T, KP>(row, u));
                Pk<T> p = Pk<T>::ld(a.P + boff<T, KP>(row, u));
#pragma unroll
                for (int q = 0; q < L; ++q)
                    if (s_act[u * L + q])
                        p.v[q] = first ? r.v[q] : fma(s_coef[u * L + q], p.v[q], r.v[q]);
                p.st(a.P + boff<T, KP>(row, u));
                group_fence();
            }
        }
        wred_zero();
        if (!barrier()) {
            finish(false);
            return;
        }
        if (stats_thread) tally.begin();

        // ---------------- phase 2: w = S p, p^T w
        {
            bool ga[G];
#pragma unroll
            for (int u = 0; u < G; ++u) ga[u] = s_gact[u] != 0;
            // FP32, while every group is active: two entries' loads in flight per
            // lane instead of one's (30 steps, one entry against two: 64^3 27-point
            // k = 8 1335 and 1066 us, k = 28 4071 and 3452; 72^3 7-point 774 and 768,
            // 3596 and 3398).  At 16 and 20 columns the 64 registers are few for the
            // loads, and the operator decides: 700^2 5-point k = 16 1954 and 2014 us,
            // k = 20 2633 and 2721; 72^3 7-point 1551 and 1581, 2100 and 2116; 64^3
            // 27-point 2068 and 2020, 2467 and 2354; 128^3 7-point k = 20 12.5 and 11.7
            // ms.  Operators of few entries per row are the common ones: one entry.
            // Not in FP64, which its FMAs bound.
            constexpr bool two_entries = sizeof(T) == 4 && (KP < 16 || KP > 20);
            bool all_active = true;
#pragma unroll
            for (int u = 0; u < G; ++u) all_active &= ga[u];
            for (int s = s0 + warp; s < s1; s += nwarps) {
                const long long beg = a.sp[s], end = a.sp[s + 1];
                const int width = (int)((end - beg) >> 5);
                if constexpr (kSplitGather<T, KP>) {
                    // one half of the column groups of a slice's rows: w, then the
                    // partial sums of p^T w over those columns
                    auto spmm_half = [&](auto half_tag, int s, int width, long long e0) {
                        constexpr int H = decltype(half_tag)::value;
                        constexpr int NU = G / 2, U0 = H * NU;
                        T acc[NU * L];
#pragma unroll
                        for (int c = 0; c < NU * L; ++c) acc[c] = T(0);
                        gather_row_part<T, KP, U0, NU>(a.col, a.val, e0, width, a.P, acc);
                        const int row = s * 32 + lane;
#pragma unroll
                        for (int u = 0; u < NU; ++u) {
                            if (!ga[U0 + u] || row >= n) {
#pragma unroll
                                for (int q = 0; q < L; ++q) acc[u * L + q] = T(0);
                                continue;
                            }
                            Pk<T> w;
#pragma unroll
                            for (int q = 0; q < L; ++q) w.v[q] = acc[u * L + q];
                            w.st(a.W + boff<T, KP>(row, U0 + u));
                            const Pk<T> p = Pk<T>::ld(a.P + boff<T, KP>(row, U0 + u));
#pragma unroll
                            for (int q = 0; q < L; ++q)
                                acc[u * L + q] = s_act[(U0 + u) * L + q] ? p.v[q] * w.v[q] : T(0);
                        }
                        warp_cols_add<T, NU * L>(acc, wred[warp] + U0 * L, lane);
                    };
                    spmm_half(std::integral_constant<int, 0>{}, s, width, beg + lane);
                    spmm_half(std::integral_constant<int, 1>{}, s, width, beg + lane);
                } else {
                    T acc[KP];
#pragma unroll
                    for (int c = 0; c < KP; ++c) acc[c] = T(0);
                    if (two_entries && all_active)
                        gather_row_part<T, KP, 0, G>(a.col, a.val, beg + lane, width, a.P, acc);
                    else
                        gather_row<T, KP>(a.col, a.val, beg + lane, width, a.P, ga, acc);
                    const int row = s * 32 + lane;
                    if (row < n) {
#pragma unroll
                        for (int u = 0; u < G; ++u) {
                            if (!ga[u]) continue;
                            Pk<T> w;
#pragma unroll
                            for (int q = 0; q < L; ++q) w.v[q] = acc[u * L + q];
                            w.st(a.W + boff<T, KP>(row, u));
                            const Pk<T> p = Pk<T>::ld(a.P + boff<T, KP>(row, u));
#pragma unroll
                            for (int q = 0; q < L; ++q)
                                acc[u * L + q] = s_act[u * L + q] ? p.v[q] * w.v[q] : T(0);
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < KP; ++c) acc[c] = T(0);
                    }
#pragma unroll
                    for (int u = 0; u < G; ++u)
                        if (!ga[u]) {
#pragma unroll
                            for (int q = 0; q < L; ++q) acc[u * L + q] = T(0);
                        }
                    warp_cols_add<T, KP>(acc, wred[warp], lane);
                }
            }
            publish(0);
        }
        if (!barrier()) {
            finish(false);
            return;
        }
        // alpha = rho / p^T w (src/ops_lin_sol.c:300-330)
        total(0, [&](int c, double ptw) {
            if (c >= k) {
                s_coef[c] = T(0);
                return;
            }
            const double rho = sc->rho2[c];
            const double al = s_act[c] ? scalar_quotient<T>(rho, ptw) : 0.0;
            sc->ptw[c] = ptw;
            sc->rho1[c] = rho;
            sc->alpha[c] = al;
            s_coef[c] = (T)al;
        });
        if (stats_thread) {
            int gact = 0;
            for (int u = 0; u < G; ++u) gact += s_gact[u];
            tally.end(gact);
        }

        // ---------------- phase 3: x += alpha p, r -= alpha w, r^T r
        wred_zero();  // (synchronises the block)
        for_parts([&](auto part) {
            constexpr int U0 = decltype(part)::value * GP;
            T racc[KPP];
#pragma unroll
            for (int c = 0; c < KPP; ++c) racc[c] = T(0);
            for (int row = r0 + tid; row < r1; row += kPcgThreads) {
#pragma unroll
                for (int uu = 0; uu < GP; ++uu) {
                    const int u = U0 + uu;
                    if (!s_gact[u]) continue;
                    Pk<T> x = Pk<T>::ld(a.X + boff<T, KP>(row, u));
                    Pk<T> r = Pk<T>::ld(a.R + boff<T, KP>(row, u));
                    const Pk<T> p = Pk<T>::ld(a.P + boff<T, KP>(row, u));
                    const Pk<T> w = Pk<T>::ld(a.W + boff<T, KP>(row, u));
#pragma unroll
                    for (int q = 0; q < L; ++q) {
                        const int c = u * L + q;
                        if (s_act[c]) {
                            const T al = s_coef[c];
                            x.v[q] = fma(al, p.v[q], x.v[q]);
                            r.v[q] = fma(-al, w.v[q], r.v[q]);
                            racc[uu * L + q] = fma(r.v[q], r.v[q], racc[uu * L + q]);
                        }
                    }
                    x.st(a.X + boff<T, KP>(row, u));
                    r.st(a.R + boff<T, KP>(row, u));
                    group_fence();
                }
            }
            warp_cols_add<T, KPP>(racc, wred[warp] + U0 * L, lane);
        });
        publish(0);
        if (!barrier()) {
            finish(false);
            return;
        }
        // convergence test of src/ops_lin_sol.c:383-394, on squares, and beta for
        // the next step
        int leave = -1;
        total(0, [&](int c, double rr) {
            if (c >= k || !s_act[c]) return;
            const double be = scalar_quotient<T>(rr, sc->rho1[c]);
            sc->rho2[c] = rr;
            sc->beta[c] = be;
            s_coef[c] = (T)be;
            if (!(rr > stop[c])) {
                sc->active[c] = 0;
                sc->left_at[c] = it + 1;
                leave = c;
            }
        });
        const int left = __syncthreads_count(leave >= 0);
        if (leave >= 0) s_act[leave] = 0;
        if (tid == 0) {
            s_nactive -= left;
            sc->nactive = s_nactive;
            sc->niter = it + 1;
        }
        __syncthreads();
    }
    finish(true);
}

// ---------------------------------------------------------------- small operators
// The same block CG for operators whose step is a chain of latencies rather
// than bytes or FMAs: phases of a microsecond between barriers.
//
// Work unit: one slice (32 rows, a row per lane) times one chunk of GU (one or
// two) 16-byte column groups, so that a narrow operator still fills the warps
// (an FP64 FMA occupies a scheduler for 64 clocks: 20 FP64 columns in one warp
// per slice took 42 us a step at n = 4160).  A warp keeps its U units for the
// whole solve with their x, r, p and w in registers; global memory holds only
// what other units gather.  Every block sums the partials of all blocks itself
// and keeps its own scalars, in shared memory, as are the block's matrix
// entries where they fit.
//
// FUSE (two phases, two barriers a step): a gather forms p = r + beta p of each
// neighbour as it reads r and p, and the own rows' p is stored with r after the
// alpha barrier.  Otherwise (FP64 operators with enough entries per row that
// the gather's second FMA costs more than a barrier): p is stored first, and
// gathered after a barrier of its own.  CL: the blocks are one thread-block
// cluster, its hardware barrier replaces the grid's, and every block puts its
// partial sums into the others' shared memory.
//
constexpr int kSmallThreads = 512;
constexpr int kSmallCluster = 16;          // blocks of the cluster form at most
constexpr int kSmallSmemMax = 160 * 1024;  // the rest stays L1
// Element offset of row i, 16-byte group u of a slice-blocked block of G groups
// (a small operator's blocks have fewer than 2^31 elements).
template <typename T>
__device__ __forceinline__ unsigned goff(int i, int u, int G) {
    constexpr unsigned L = Pk<T>::L;
    return (((unsigned)i >> 5) * (unsigned)G + (unsigned)u) * (32u * L) + ((unsigned)i & 31u) * L;
}

// acc += N entries (col[0], col[32], ..) of the lane's row, of which `left` are
// its own, times the groups [u0, u0 + GU) of V, or with RP of V + beta Vp.  An
// entry past the last one repeats its loads only; a group past the last one
// repeats it, and its sums are not used.
template <typename T, int GU, int N, bool RP>
__device__ __forceinline__ void unit_entries(const int *col, const T *val, int left, const T *V,
                                             const T *Vp, const T *beta, int u0, int G,
                                             T (&acc)[GU * Pk<T>::L]) {
    constexpr int L = Pk<T>::L;
    int j[N];
    T m[N];
#pragma unroll
    for (int d = 0; d < N; ++d) {
        const int dd = min(d, left - 1);
        j[d] = col[32 * dd];
        m[d] = val[32 * dd];
    }
    Pk<T> q0[N][GU], q1[N][GU];
#pragma unroll
    for (int d = 0; d < N; ++d) {
#pragma unroll
        for (int g = 0; g < GU; ++g) {
            const unsigned o = goff<T>(j[d], g == 0 ? u0 : min(u0 + g, G - 1), G);
            q0[d][g] = Pk<T>::ld(V + o);
            if constexpr (RP) q1[d][g] = Pk<T>::ld(Vp + o);
        }
    }
#pragma unroll
    for (int d = 0; d < N; ++d) {
        if (d >= left) continue;  // the same for the whole warp
#pragma unroll
        for (int g = 0; g < GU; ++g) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
                T y = q0[d][g].v[l];
                if constexpr (RP) y = fma(beta[g * L + l], q1[d][g].v[l], y);
                acc[g * L + l] = fma(m[d], y, acc[g * L + l]);
            }
        }
    }
}
template <typename T, int GU, int NE, bool RP>
__device__ __forceinline__ void unit_gather(const int *col, const T *val, int width, const T *V,
                                            const T *Vp, const T *sbeta, int u0, int G,
                                            T (&acc)[GU * Pk<T>::L]) {
    constexpr int CC = GU * Pk<T>::L;
    T beta[CC];
#pragma unroll
    for (int c = 0; c < CC; ++c) {
        acc[c] = T(0);
        beta[c] = RP ? sbeta[c] : T(0);
    }
#pragma unroll 1
    for (int e = 0; e < width; e += NE)
        unit_entries<T, GU, NE, RP>(col + 32 * e, val + 32 * e, width - e, V, Vp, beta, u0, G, acc);
}

template <typename T, int GU, int U, bool CL, bool FUSE>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_pcg_small(PcgArgs<T> a, int kp, int smem_bytes) {
    constexpr int L = Pk<T>::L, CC = GU * L;
    constexpr int NW = kSmallThreads / 32;
    // matrix entries in flight per lane (a 5- or 7-point row in one go)
    constexpr int NE = U * GU == 1 ? (sizeof(T) == 8 && FUSE ? 5 : 8)
                       : U * GU == 4 && FUSE ? 1
                                             : 8 / (U * GU * (FUSE ? 2 : 1));
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ T wred[NW * U][CC];  // column sums of each unit
    __shared__ double sums[2][kPcgMaxCols];
    __shared__ double stop[kPcgMaxCols];  // r^T r at which a column leaves
    // the partial sums of every block of the cluster, two sets of two; else the
    // column sums of each stripe
    __shared__ double stripe[CL ? 4 * kSmallCluster * kPcgMaxCols : kSmallThreads];
    __shared__ T s_alpha[kPcgMaxCols], s_beta[kPcgMaxCols];
    __shared__ int s_act[kPcgMaxCols];
    __shared__ int s_nactive;
    __shared__ PcgScalars s_sc;
    PcgScalars *sc = &s_sc;
    PcgSync *gs = a.sync;
    int *error = &a.sync->error;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = a.k, n = a.n, G = kp / L, nch = (G + GU - 1) / GU;
    const int nb = gridDim.x, me = blockIdx.x;
    const bool stats_thread = me == 0 && tid == kSmallThreads - 1;
    __shared__ PcgTally<T> tally;
    if (stats_thread) tally.clear();
    if (!CL && a.withhold_last && nb > 1 && me == nb - 1) return;
    if constexpr (CL) cooperative_groups::this_cluster().sync();  // all blocks run

    const int s0 = (int)((long long)a.nslices * me / nb);
    const int s1 = (int)((long long)a.nslices * (me + 1) / nb);
    const int nsl = s1 - s0;  // nsl nch <= U NW by the launch's choice
    // the block's matrix entries in shared memory where they fit
    const long long e_lo = a.sp[s0], e_cnt = a.sp[s1] - e_lo;
    const bool in_smem = e_cnt * (long long)(sizeof(T) + 4) <= smem_bytes;
    T *sval = reinterpret_cast<T *>(dsm);
    int *scol = reinterpret_cast<int *>(sval + (in_smem ? e_cnt : 0));
    if (in_smem) {
        for (int i = tid; i < (int)e_cnt; i += kSmallThreads) {
            sval[i] = a.val[e_lo + i];
            scol[i] = a.col[e_lo + i];
        }
    }
    for (int c = tid; c < kPcgMaxCols; c += kSmallThreads) {
        s_act[c] = 0;
        s_alpha[c] = s_beta[c] = T(0);
    }
    __syncthreads();

    // this warp's units
    int slice[U], u0[U], width[U], ent[U];
    bool live[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
        const int v = warp + i * NW;
        live[i] = v < nsl * nch;
        slice[i] = live[i] ? s0 + v / nch : s0;
        u0[i] = live[i] ? (v % nch) * GU : 0;
        const long long beg = live[i] ? a.sp[slice[i]] : 0, end = live[i] ? a.sp[slice[i] + 1] : 0;
        width[i] = (int)((end - beg) >> 5);
        ent[i] = (int)(beg - e_lo) + lane;
    }
    auto has_row = [&](int i) { return slice[i] * 32 + lane < n; };
    T x[U][CC], r[U][CC], p[U][CC], w[U][CC];

    // w = the unit's rows of S V, and of S (R + beta P)
    auto gather = [&](int i, const T *V, T (&acc)[CC]) {
        if (in_smem)
            unit_gather<T, GU, NE, false>(scol + ent[i], sval + ent[i], width[i], V, V, s_beta, u0[i],
                                      G, acc);
        else
            unit_gather<T, GU, NE, false>(a.col + e_lo + ent[i], a.val + e_lo + ent[i], width[i], V, V,
                                      s_beta, u0[i], G, acc);
    };
    auto gather_rp = [&](int i, T (&acc)[CC]) {
        if (in_smem)
            unit_gather<T, GU, NE, true>(scol + ent[i], sval + ent[i], width[i], a.R, a.P,
                                     s_beta + u0[i] * L, u0[i], G, acc);
        else
            unit_gather<T, GU, NE, true>(a.col + e_lo + ent[i], a.val + e_lo + ent[i], width[i], a.R,
                                     a.P, s_beta + u0[i] * L, u0[i], G, acc);
    };
    auto store = [&](T *v, int i, const T (&q)[CC]) {
#pragma unroll
        for (int g = 0; g < GU; ++g)
            if (u0[i] + g < G && has_row(i)) {
                Pk<T> o;
#pragma unroll
                for (int l = 0; l < L; ++l) o.v[l] = q[g * L + l];
                o.st(v + goff<T>(slice[i] * 32 + lane, u0[i] + g, G));
            }
    };
    auto load = [&](const T *v, int i, T (&q)[CC]) {
#pragma unroll
        for (int g = 0; g < GU; ++g) {
            const bool in = live[i] && u0[i] + g < G && has_row(i);
            Pk<T> o;
            if (in) o = Pk<T>::ld(v + goff<T>(slice[i] * 32 + lane, u0[i] + g, G));
#pragma unroll
            for (int l = 0; l < L; ++l) q[g * L + l] = in ? o.v[l] : T(0);
        }
    };
    // column sums of q over the unit's rows, into its row of wred
    auto unit_sum = [&](int i, T (&q)[CC]) {
        const T s = warp_cols_reduce<T, CC>(q, lane);
        if (lane < CC) wred[warp + i * NW][lane] = s;
    };
    // Two sets of partials alternate by the barrier's parity: blocks read them
    // after a barrier while faster ones already write the next phase's, and a set
    // is rewritten only after the following barrier.
    unsigned long long epoch = 0;
    auto part_of = [&](unsigned long long e, int which) {
        return a.part + ((size_t)(e & 1) * 2 + which) * nb * kp;
    };
    // this block's column sums of wred, for the next barrier: into the other
    // blocks' shared memory in a cluster, else into global memory
    auto publish = [&](int which) {
        __syncthreads();
        lane_cols_sum(
            kp, nsl, [&](int sl, int c) { return (double)wred[sl * nch + c / CC][c % CC]; },
            [&](int c, double t, int q) {
                if constexpr (CL) {
                    double *at = stripe + ((((epoch + 1) & 1) * 2 + which) * nb + me) * kp + c;
                    for (int b = q; b < nb; b += kp <= 16 ? 8 : 4)
                        *cooperative_groups::this_cluster().map_shared_rank(at, b) = t;
                } else if (q == 0) {
                    part_of(epoch + 1, which)[(size_t)me * kp + c] = t;
                }
            });
    };
    // sums of the partials over the blocks; the caller synchronises the block
    auto total = [&](int which, auto use) {
        if constexpr (CL) {
            const double *part = stripe + ((epoch & 1) * 2 + which) * nb * kp;
            lane_cols_sum(
                kp, nb, [&](int b, int c) { return part[b * kp + c]; },
                [&](int c, double t, int q) {
                    if (q == 0) use(c, t);
                });
        } else {
            grid_cols_sum<kSmallThreads>(part_of(epoch, which), nb, kp, stripe, use);
        }
    };
    auto barrier = [&]() {
        ++epoch;
        if constexpr (CL) {
            cooperative_groups::this_cluster().sync();
            return true;
        } else {
            return grid_arrive_wait(gs, error, a.timeout_ns, a.max_polls, epoch);
        }
    };
    auto finish = [&](bool ok) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < U; ++i)
            if (live[i]) store(a.X, i, x[i]);
        if constexpr (sizeof(T) == 4) {  // columns of x that left FP32's range
            unsigned long long out = 0;
#pragma unroll
            for (int i = 0; i < U; ++i)
#pragma unroll
                for (int c = 0; c < CC; ++c)
                    if (live[i] && has_row(i) && !isfinite(x[i][c])) out |= 1ull << (u0[i] * L + c);
            if (out) atomicOr(&gs->out_of_range, out);
        }
        if (me == 0) {  // the host reads the first block's scalars
            if (tid < k) sc->last_res[tid] = sqrt(sc->rho2[tid]);
            __syncthreads();
            const int *src = reinterpret_cast<const int *>(sc);
            int *dst = reinterpret_cast<int *>(a.sc);
            for (int i = tid; i < (int)(sizeof(PcgScalars) / sizeof(int)); i += kSmallThreads)
                dst[i] = src[i];
        }
        if (me == 0 && tid == 0) {
            if (!ok || *(volatile int *)error) a.stats->error = 1;
            a.stats->launches += 1;
            a.stats->iters += (unsigned long long)sc->niter;
        }
        if (stats_thread) tally.write(a, kp);
    };

    // ---------------- r = b - S x (or r = b for x = 0), p = 0, norms
#pragma unroll
    for (int i = 0; i < U; ++i) {
        T b[CC], q[CC];
        load(a.B, i, b);
        if (a.x_zero) {
#pragma unroll
            for (int c = 0; c < CC; ++c) x[i][c] = w[i][c] = T(0);
        } else {
            load(a.X, i, x[i]);
            if (live[i]) gather(i, a.X, w[i]);
        }
#pragma unroll
        for (int c = 0; c < CC; ++c) {
            p[i][c] = T(0);
            r[i][c] = live[i] && has_row(i) ? (a.x_zero ? b[c] : b[c] - w[i][c]) : T(0);
            q[c] = r[i][c] * r[i][c];
        }
        if (live[i]) {
            if constexpr (FUSE) {
                store(a.R, i, r[i]);
                store(a.P, i, p[i]);
            }
            unit_sum(i, q);
        }
    }
    publish(0);
    if (a.rel_tol) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < U; ++i) {
            T b[CC];
            load(a.B, i, b);
#pragma unroll
            for (int c = 0; c < CC; ++c) b[c] = b[c] * b[c];
            if (live[i]) unit_sum(i, b);
        }
        publish(1);
    }
    if (!barrier()) {
        if (tid == 0) sc->niter = 0;
        finish(false);
        return;
    }
    // initial residual norms (src/ops_lin_sol.c:171-233)
    total(0, [&](int c, double t) { sums[0][c] = t; });
    if (a.rel_tol) {
        __syncthreads();
        total(1, [&](int c, double t) { sums[1][c] = t; });
    }
    __syncthreads();
    if (tid < kPcgMaxCols) {
        const int c = tid;
        int on = 0;
        if (c < k) {
            const double nrm = a.rel_tol ? sqrt(sums[1][c]) : 1.0;
            const double rr = sums[0][c], res = sqrt(rr);
            sc->norm_b[c] = nrm;
            sc->rho2[c] = rr;
            sc->init_res[c] = res;
            sc->last_res[c] = res;
            sc->beta[c] = 0.0;
            sc->alpha[c] = 0.0;
            on = res > a.tol * nrm ? 1 : 0;
            stop[c] = stop_square(a.rate * res, a.tol * nrm);
        }
        sc->active[c] = s_act[c] = on;
        sc->left_at[c] = 0;
    }
    __syncthreads();
    if (tid == 0) {
        int cnt = 0;
        for (int c = 0; c < k; ++c) cnt += s_act[c];
        s_nactive = sc->nactive = cnt;
        sc->niter = 0;
    }
    __syncthreads();

    for (int it = 0; it < a.max_iter && s_nactive > 0; ++it) {
        // units none of whose columns is active rest
        bool act[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
            int any = 0;
#pragma unroll
            for (int c = 0; c < CC; ++c) any |= s_act[u0[i] * L + c];
            act[i] = live[i] && any != 0;
        }
        // ---------------- p = r + beta p
#pragma unroll
        for (int i = 0; i < U; ++i)
            if (act[i]) {
#pragma unroll
                for (int c = 0; c < CC; ++c)
                    if (s_act[u0[i] * L + c]) p[i][c] = fma(s_beta[u0[i] * L + c], p[i][c], r[i][c]);
                if constexpr (!FUSE) store(a.P, i, p[i]);
            }
        if constexpr (!FUSE) {
            if (!barrier()) {
                finish(false);
                return;
            }
        }
        if (stats_thread) tally.begin();
        // ---------------- w = S p, p^T w
#pragma unroll
        for (int i = 0; i < U; ++i) {
            T q[CC];
#pragma unroll
            for (int c = 0; c < CC; ++c) q[c] = T(0);
            if (act[i]) {
                if constexpr (FUSE) gather_rp(i, w[i]);
                else gather(i, a.P, w[i]);
#pragma unroll
                for (int c = 0; c < CC; ++c)
                    q[c] = s_act[u0[i] * L + c] && has_row(i) ? p[i][c] * w[i][c] : T(0);
            }
            if (live[i]) unit_sum(i, q);
        }
        publish(0);
        if (!barrier()) {
            finish(false);
            return;
        }
        // alpha = rho / p^T w (src/ops_lin_sol.c:300-330)
        total(0, [&](int c, double ptw) {
            if (c >= k) return;
            const double rho = sc->rho2[c];
            const double al = s_act[c] ? scalar_quotient<T>(rho, ptw) : 0.0;
            sc->ptw[c] = ptw;
            sc->rho1[c] = rho;
            sc->alpha[c] = al;
            s_alpha[c] = (T)al;
        });
        if (stats_thread) {
            int gact = 0;
            for (int u = 0; u < G; ++u) {
                int any = 0;
                for (int l = 0; l < L; ++l) any |= s_act[u * L + l];
                gact += any != 0;
            }
            tally.end(gact);
        }
        __syncthreads();
        // ---------------- x += alpha p, r -= alpha w, r^T r
#pragma unroll
        for (int i = 0; i < U; ++i) {
            T q[CC];
#pragma unroll
            for (int c = 0; c < CC; ++c) {
                q[c] = T(0);
                if (act[i] && s_act[u0[i] * L + c]) {
                    const T al = s_alpha[u0[i] * L + c];
                    x[i][c] = fma(al, p[i][c], x[i][c]);
                    r[i][c] = fma(-al, w[i][c], r[i][c]);
                    q[c] = has_row(i) ? r[i][c] * r[i][c] : T(0);
                }
            }
            if constexpr (FUSE) {
                if (act[i]) {
                    store(a.R, i, r[i]);
                    store(a.P, i, p[i]);
                }
            }
            if (live[i]) unit_sum(i, q);
        }
        publish(0);
        if (!barrier()) {
            finish(false);
            return;
        }
        // convergence test of src/ops_lin_sol.c:383-394, on squares, and beta for
        // the next step
        int leave = -1;
        total(0, [&](int c, double rr) {
            if (c >= k || !s_act[c]) return;
            const double be = scalar_quotient<T>(rr, sc->rho1[c]);
            sc->rho2[c] = rr;
            sc->beta[c] = be;
            s_beta[c] = (T)be;
            if (!(rr > stop[c])) {
                sc->active[c] = 0;
                sc->left_at[c] = it + 1;
                leave = c;
            }
        });
        const int left = __syncthreads_count(leave >= 0);
        if (leave >= 0) s_act[leave] = 0;
        if (tid == 0) {
            s_nactive -= left;
            sc->nactive = s_nactive;
            sc->niter = it + 1;
        }
        __syncthreads();
    }
    finish(true);
}

// Cluster size the cluster form may have (16 CTAs where the device schedules
// such a cluster, else 8), or 0 when neither can run.
template <typename T, int GU, int U>
int pcg_small_cluster() {
    static PerDevice<int> cache;
    return cache.get([] {
        auto *kern = k_pcg_small<T, GU, U, true, true>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kSmallSmemMax) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        for (int c : {kSmallCluster, 8}) {
            if (c > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                              1) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(kSmallThreads);
            cfg.dynamicSmemBytes = kSmallSmemMax;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = c;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            if (nc > 0) return c;
        }
        return 0;
    });
}

template <typename T, int GU, int U, bool FUSE>
void launch_pcg_small_form(const PcgArgs<T> &a, int kp, bool cluster, int nb, cudaStream_t st) {
    // room for a block's matrix entries, a quarter more than an even share; a
    // block with more reads them from global memory
    const double share = 1.25 * (double)a.stored / nb * (sizeof(T) + 4.0) + 4096.0;
    const int smem = (int)std::min((double)kSmallSmemMax, share) & ~15;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (FUSE && cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = nb;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        GCGE_CUDA(cudaLaunchKernelEx(&cfg, k_pcg_small<T, GU, U, true, true>, a, kp, smem));
    } else {
        static PerDevice<bool> smem_set;
        smem_set.get([] {
            GCGE_CUDA(cudaFuncSetAttribute(k_pcg_small<T, GU, U, false, FUSE>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kSmallSmemMax));
            return true;
        });
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        GCGE_CUDA(cudaLaunchKernelEx(&cfg, k_pcg_small<T, GU, U, false, FUSE>, a, kp, smem));
    }
    count_launch();
}

// Runs the solve in k_pcg_small where the units of its operator fit the warps
// (two each); false where they do not, and the three-phase grid kernel takes it.
// Measured, us per step of a 30-step solve, three-phase kernel (or its former
// cluster form) -> this one:
//   5-point n = 4160    k = 4 FP32 9.3 -> 4.6, FP64 16 -> 8.8; k = 20 FP64 37 -> 11.9
//   5-point n = 16384   k = 4 FP32 13 -> 7.8, FP64 24 -> 9.7; k = 20 27 -> 10.5, 38 -> 21.1
//   7-point 32^3        k = 4 FP32 22 -> 8.4, FP64 26 -> 13.0; k = 20 FP32 29 -> 15.2
//   27-point 24^3       k = 20 FP32 36 -> 13.3, FP64 59 -> 28.3
// Most of a short step is not the gather but the FP64 scalars: with a block-wide
// tree over every block's partials, a division and a square root a step took
// 7.3 us at n = 4160, k = 4 FP32 (7.3 -> 4.6; n = 16384 10.3 -> 7.8; 27-point 24^3,
// k = 20 14.7 -> 13.3).
// FUSE: the gather's second vector against a barrier.  In FP64 its FMAs decide
// (entries k / 2 clocks over the SMs; 5-point k = 20, n = 7400: 16.8 us both at
// 2429, k = 12 14.1 against 14.8 at 1458, k = 40 26.2 against 24.5 at 4859), in
// FP32 its loads (27-point 24^3, k = 20 15.1 against 15.3 at 23900, k = 40 20.0
// against 18.4 at 47700).
// Cluster or grid: the cluster's barriers are shorter and its partials stay in
// shared memory, but it has 16 of the 152 SMs.  FP32, cluster against grid: with
// a unit per warp 5-point n = 7400, k = 8 (2300 clocks) 6.1 against 8.1 us, 7-point
// 20^3, k = 8 (3500) 6.7 against 8.0; with two, n = 4160, k = 12 (1950) 7.7
// against 8.3, n = 16384, k = 4 (2560) 8.8 against 7.8, n = 7400, k = 12 (3470) 8.9
// against 8.7.  FP64 n = 4160, k = 4 (7800) 9.6 against 8.8.
template <typename T>
constexpr double kFuseClocks = sizeof(T) == 8 ? 2200.0 : 30000.0;
template <typename T>
constexpr double cluster_clocks(bool one_unit) {
    return sizeof(T) == 8 ? 6000.0 : one_unit ? 4000.0 : 2000.0;
}
template <typename T>
bool launch_pcg_small(const PcgArgs<T> &a, int kp, cudaStream_t st) {
    constexpr int NW = kSmallThreads / 32;
    const int G = kp / Pk<T>::L;
    const int sms = std::max(1, device_sms() / std::max(1, t_pcg_share));
    const double entries = (double)a.stored * kp;
    const bool fuse = entries / 2.0 / sms < kFuseClocks<T>;
    // clocks of a step over all SMs: FP64 FMAs (two per clock), or gathered bytes
    // (64 per clock)
    const double work = sizeof(T) == 8 ? (2.0 * entries + 5.0 * a.n * kp) / 2.0
                                       : 2.0 * entries * sizeof(T) / 64.0;
    auto units = [&](int nb, int gu) { return (a.nslices + nb - 1) / nb * ((G + gu - 1) / gu); };
    const int csize = std::min(pcg_small_cluster<T, 1, 1>(),
                               std::min(pcg_small_cluster<T, 2, 1>(), pcg_small_cluster<T, 2, 2>()));
    const bool cluster =
        fuse && csize > 0 && units(csize, 2) <= 2 * NW &&
        work / csize <= cluster_clocks<T>(units(csize, 2) <= NW);
    const int nb = cluster ? csize : std::max(1, std::min(sms, a.nslices));
    if (!cluster && units(nb, 2) > 2 * NW) return false;
    t_pcg_form = cluster ? kPcgCluster : kPcgUnits;
    // narrow chunks while every warp has one unit at most: more warps at work
    const int gu = units(nb, 1) <= NW ? 1 : 2, u = units(nb, gu) <= NW ? 1 : 2;
    auto go = [&](auto GU, auto U) {
        constexpr int g = decltype(GU)::value, v = decltype(U)::value;
        if (fuse) launch_pcg_small_form<T, g, v, true>(a, kp, cluster, nb, st);
        else launch_pcg_small_form<T, g, v, false>(a, kp, cluster, nb, st);
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    if (gu == 1) go(One{}, One{});
    else if (u == 1) go(Two{}, One{});
    else go(Two{}, Two{});
    return true;
}

template <typename T, int KP>
void launch_block_pcg(PcgArgs<T> a, cudaStream_t st) {
    static PerDevice<bool> fits;
    GCGE_REQUIRE(fits.get([] {
        int b = 0;
        GCGE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_block_pcg<T, KP>,
                                                                pcg_threads<T, KP>(), 0));
        return b >= 1;
    }),
                 GCGE_ERR_CUDA, "block PCG: kernel does not fit on an SM");
    const int nb = std::max(1, std::min(device_sms() / std::max(1, t_pcg_share), a.nslices));
    t_pcg_form = kPcgPhases;
    void *args[] = {&a};
    GCGE_CUDA(cudaLaunchCooperativeKernel((const void *)k_block_pcg<T, KP>, dim3(nb),
                                          dim3(pcg_threads<T, KP>()), args, 0, st));
    count_launch();
}

}  // namespace

template <typename T>
void block_pcg_rows(PcgWork &wk, const SellPattern &pat, const T *sval, const T *Bv, T *X, T *R,
                    T *P, T *W, int kp, int k, int max_iter, double rate, double tol, bool rel_tol,
                    bool x_zero, cudaStream_t st) {
    constexpr int L = 16 / (int)sizeof(T);
    GCGE_REQUIRE(k >= 1 && k <= kp && kp <= 40 && kp % L == 0 && k <= kPcgMaxCols, GCGE_ERR_ARG,
                 "block_pcg: block width");
    if (pat.n == 0) return;
    PcgArgs<T> a;
    a.sp = pat.slice_ptr.p;
    a.col = pat.col.p;
    a.val = sval;
    a.n = pat.n;
    a.nslices = pat.nslices;
    a.stored = pat.padded;
    a.B = Bv;
    a.X = X;
    a.R = R;
    a.P = P;
    a.W = W;
    a.k = k;
    a.max_iter = std::max(0, max_iter);
    a.rel_tol = rel_tol ? 1 : 0;
    a.x_zero = x_zero ? 1 : 0;
    a.rate = rate;
    a.tol = tol;
    a.matrix_bytes = (double)pat.nnz * (sizeof(T) + 4) + 4.0 * (pat.n + 1);
    a.sc = wk.sc.p;
    a.sync = wk.sync.p;
    a.stats = wk.stats.p;
    a.part = wk.part.p;
    a.timeout_ns = kBarrierTimeoutNs;
    a.max_polls = kBarrierMaxPolls;
    a.withhold_last = 0;
    if (t_pcg_barrier_test.active) {
        a.timeout_ns = t_pcg_barrier_test.timeout_ns;
        a.withhold_last = t_pcg_barrier_test.withhold_last;
    }
    GCGE_CUDA(cudaMemsetAsync(wk.sync.p, 0, sizeof(PcgSync), st));
    const bool timed = wk.ev_used + 2 <= 65536;
    if (timed) {
        while (wk.ev.size() < wk.ev_used + 2) {
            cudaEvent_t e;
            GCGE_CUDA(cudaEventCreate(&e));
            wk.ev.push_back(e);
        }
        GCGE_CUDA(cudaEventRecord(wk.ev[wk.ev_used], st));
    }
    if (launch_pcg_small<T>(a, kp, st)) {
        // (small operators; their kernel marks the columns out of range itself)
    } else if constexpr (sizeof(T) == 4) {
        switch (kp) {
#define GCGE_PCG_CASE(W_)                                     \
    case W_:                                                  \
        launch_block_pcg<T, W_>(a, st);                       \
        break;
            GCGE_PCG_CASE(4) GCGE_PCG_CASE(8) GCGE_PCG_CASE(12) GCGE_PCG_CASE(16)
            GCGE_PCG_CASE(20) GCGE_PCG_CASE(24) GCGE_PCG_CASE(28) GCGE_PCG_CASE(32)
            GCGE_PCG_CASE(36) GCGE_PCG_CASE(40)
            default: throw CudaError{GCGE_ERR_ARG, "block_pcg: unsupported width"};
        }
    } else {
        switch (kp) {
            GCGE_PCG_CASE(2) GCGE_PCG_CASE(4) GCGE_PCG_CASE(6) GCGE_PCG_CASE(8)
            GCGE_PCG_CASE(12) GCGE_PCG_CASE(16) GCGE_PCG_CASE(20) GCGE_PCG_CASE(24)
            GCGE_PCG_CASE(28) GCGE_PCG_CASE(32) GCGE_PCG_CASE(36) GCGE_PCG_CASE(40)
#undef GCGE_PCG_CASE
            default: throw CudaError{GCGE_ERR_ARG, "block_pcg: unsupported width"};
        }
    }
    if (timed) {
        GCGE_CUDA(cudaEventRecord(wk.ev[wk.ev_used + 1], st));
        wk.ev_used += 2;
    }
    if constexpr (sizeof(T) == 4) {  // of a correction, which starts from zero
        if (x_zero && t_pcg_form == kPcgPhases) mark_out_of_range(pat.n, kp, X, &wk.sync.p->out_of_range, st);
    }
    wk.launches++;
}

}  // namespace gcge
