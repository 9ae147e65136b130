// Dense symmetric eigensolver for the Rayleigh-Ritz projected matrix
// (replaces the reference's dsyevx call, src/ops_eig_sol_gcg.c:1145-1150 /
// :1207-1209: all eigenpairs, ascending).
//
// GB300 issues FP64 at ~1/58 of its FP32 rate, so an FP64 Jacobi on one SM
// would take tens of milliseconds for s = 200.  The solver therefore
//   1. runs a parallel-order (round-robin) two-sided cyclic Jacobi in FP32,
//      logging each round's rotations: up to s = 104 in one CTA with the matrix
//      in its shared memory, above in a cluster of 8 CTAs whose shared memories
//      hold the matrix rows of the pairs each CTA owns (distributed shared
//      memory; rows move between neighbouring CTAs as the round-robin order
//      advances; where no cluster can be placed, in one 1024-thread CTA with
//      the packed upper triangle);
//   2. rebuilds the eigenvector matrix from the rotation log with one warp
//      per row (rows of V = J_1 J_2 ... J_T are independent);
//   3. refines eigenvectors and eigenvalues to FP64 accuracy with the
//      iterative refinement of Ogita & Aishima ("Iterative refinement for
//      symmetric eigenvalue decomposition", Japan J. Indust. Appl. Math. 35,
//      2018), whose cost is four s x s FP64 products per step spread over
//      all SMs;
//   4. diagonalises each remaining cluster of nearly equal eigenvalues
//      exactly on the host (tiny FP64 Jacobi) and sorts ascending.
// The 2x2 rotation is the symmetric Schur decomposition of Golub & Van Loan
// (Matrix Computations, Alg. 8.4.1).
#include <cooperative_groups.h>
#include <mutex>
#include <algorithm>
#include <cmath>
#include <numeric>

#include "common.cuh"
#include "eig.cuh"

namespace gcge {

namespace cg = cooperative_groups;

constexpr int kJacobiThreads = 1024;
constexpr int kMaxSweeps = 12;
constexpr float kRotTol = 1e-7f;   // skip rotations below FP32 resolution
constexpr float kOffTol = 2e-6f;   // ||offdiag||_F <= kOffTol ||A||_F ends the sweeps
constexpr double kClusterGap = 1e-5;      // relative gap below which pairs are clustered
constexpr double kStrongCoupling = 1e-2;  // |E_ij| above which pairs are clustered

__host__ __device__ inline int jac_m(int s) { return (s + 1) & ~1; }

// Round-robin pair i of round r for m (even) indices: element m-1 is fixed.
__host__ __device__ inline void jac_pair(int m, int r, int i, int &p, int &q) {
    int a, b;
    if (i == 0) {
        a = m - 1;
        b = r;
    } else {
        a = (r + i) % (m - 1);
        b = (r - i + (m - 1)) % (m - 1);
    }
    p = a < b ? a : b;
    q = a < b ? b : a;
}

__device__ inline int pk(int x, int y) {  // packed upper index, x <= y
    return (y * (y + 1)) / 2 + x;
}
__device__ inline int pks(int x, int y) { return x <= y ? pk(x, y) : pk(y, x); }

size_t jacobi_smem_bytes(int s) {
    const int m = jac_m(s);
    return (size_t)s * (s + 1) / 2 * sizeof(float) + (size_t)(m / 2) * 2 * sizeof(float) +
           (size_t)(m / 2) * 2 * sizeof(short) + 64;
}
static size_t jacobi_dyn_limit();
static bool jacobi_cluster_usable();
static int jacobi_cluster_max_dim();
// one-CTA kernel capacity, and the cluster kernel's where it can run
int jacobi_max_dim() {
    const size_t lim = jacobi_dyn_limit();
    int s = 8;
    while (jacobi_smem_bytes(s + 1) <= lim) ++s;
    if (jacobi_cluster_usable()) s = std::max(s, jacobi_cluster_max_dim());
    return s;
}

__global__ void __launch_bounds__(kJacobiThreads)
k_jacobi32(int s, const double *__restrict__ M, int ldm, float4 *__restrict__ log, int max_rounds,
           int *__restrict__ info /* [0]=rounds, [1]=sweeps, [2]=converged */) {
    extern __shared__ float sm[];
    const int m = jac_m(s);
    const int np = m / 2;
    float *A = sm;
    float *cs = A + (size_t)s * (s + 1) / 2;
    float *sn = cs + np;
    short *pp = reinterpret_cast<short *>(sn + np);  // pair table of the round: p, q
    __shared__ float red_off[32], red_tot[32];
    __shared__ int stop;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = blockDim.x >> 5;
    const int nq = np + (np & 1), width = nq + 1, nblk = (nq / 2) * width;
    for (int idx = t; idx < s * (s + 1) / 2; idx += blockDim.x) {
        // decode packed index -> (x, y), x <= y
        int y = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
        while ((y + 1) * (y + 2) / 2 <= idx) ++y;
        while (y * (y + 1) / 2 > idx) --y;
        const int x = idx - y * (y + 1) / 2;
        A[idx] = (float)(0.5 * (M[x + (size_t)y * ldm] + M[y + (size_t)x * ldm]));
    }
    __syncthreads();
    int round = 0, sweep = 0, converged = 0;
    for (sweep = 0; sweep < kMaxSweeps && round + (m - 1) <= max_rounds; ++sweep) {
        // stop when the off-diagonal mass is at the FP32 noise level
        float off = 0.0f, tot = 0.0f;
        for (int idx = t; idx < s * (s + 1) / 2; idx += blockDim.x) {
            int y = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
            while ((y + 1) * (y + 2) / 2 <= idx) ++y;
            while (y * (y + 1) / 2 > idx) --y;
            const int x = idx - y * (y + 1) / 2;
            const float v = A[idx] * A[idx];
            tot += x == y ? v : 2.0f * v;
            if (x != y) off += 2.0f * v;
        }
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if (lane == 0) {
            red_off[warp] = off;
            red_tot[warp] = tot;
        }
        __syncthreads();
        if (t == 0) {
            float a = 0.f, b = 0.f;
            for (int w = 0; w < nwarps; ++w) {
                a += red_off[w];
                b += red_tot[w];
            }
            stop = (a <= kOffTol * kOffTol * b) ? 1 : 0;
        }
        __syncthreads();
        if (stop) {
            converged = 1;
            break;
        }
        for (int r = 0; r < m - 1; ++r) {
            // (a) pair table and rotation of each pair
            for (int i = t; i < np; i += blockDim.x) {
                int p, q;
                jac_pair(m, r, i, p, q);
                pp[2 * i] = (short)p;
                pp[2 * i + 1] = (short)q;
                float c = 1.0f, sv = 0.0f;
                if (q < s) {
                    const float app = A[pk(p, p)], aqq = A[pk(q, q)], apq = A[pk(p, q)];
                    const float thr = kRotTol * sqrtf(fabsf(app) * fabsf(aqq));
                    if (fabsf(apq) > thr && fabsf(apq) > 1e-30f) {
                        const float tau = (aqq - app) / (2.0f * apq);
                        const float tt = (tau >= 0.0f ? 1.0f : -1.0f) / (fabsf(tau) + hypotf(1.0f, tau));
                        c = rsqrtf(1.0f + tt * tt);
                        sv = tt * c;
                    }
                }
                cs[i] = c;
                sn[i] = sv;
            }
            __syncthreads();
            // (b) A <- J^T A J on every 2x2 block (i <= j) of the pair grid.  The
            // triangle of blocks is folded into nq / 2 rows of nq + 1 blocks (row r
            // holds pair rows r and nq - 1 - r), which the threads share evenly.
            for (int b = t; b < nblk; b += blockDim.x) {
                const int fr = b / width, fc = b - fr * width;
                int i, j;
                if (fc < nq - fr) {
                    i = fr;
                    j = fr + fc;
                } else {
                    i = nq - 1 - fr;
                    j = i + (fc - (nq - fr));
                }
                if (j >= np) continue;
                {
                    const float ci = cs[i], si = sn[i];
                    const float cj = cs[j], sj = sn[j];
                    if (si == 0.0f && sj == 0.0f) continue;
                    const int pi = pp[2 * i], qi = pp[2 * i + 1];
                    const bool qiv = qi < s;
                    const int pj = pp[2 * j], qj = pp[2 * j + 1];
                    const bool qjv = qj < s;
                    if (i == j) {
                        if (!qiv) continue;
                        const float app = A[pk(pi, pi)], aqq = A[pk(qi, qi)], apq = A[pk(pi, qi)];
                        const float t11 = ci * app - si * apq, t12 = ci * apq - si * aqq;
                        const float t21 = si * app + ci * apq, t22 = si * apq + ci * aqq;
                        A[pk(pi, pi)] = t11 * ci - t12 * si;
                        A[pk(qi, qi)] = t21 * si + t22 * ci;
                        A[pk(pi, qi)] = 0.0f;
                        continue;
                    }
                    const float a11 = A[pks(pi, pj)];
                    const float a12 = qjv ? A[pks(pi, qj)] : 0.0f;
                    const float a21 = qiv ? A[pks(qi, pj)] : 0.0f;
                    const float a22 = (qiv && qjv) ? A[pks(qi, qj)] : 0.0f;
                    const float t11 = ci * a11 - si * a21, t12 = ci * a12 - si * a22;
                    const float t21 = si * a11 + ci * a21, t22 = si * a12 + ci * a22;
                    A[pks(pi, pj)] = t11 * cj - t12 * sj;
                    if (qjv) A[pks(pi, qj)] = t11 * sj + t12 * cj;
                    if (qiv) A[pks(qi, pj)] = t21 * cj - t22 * sj;
                    if (qiv && qjv) A[pks(qi, qj)] = t21 * sj + t22 * cj;
                }
            }
            // (c) log the round
            for (int i = t; i < np; i += blockDim.x)
                log[(size_t)round * np + i] = make_float4(cs[i], sn[i], __int_as_float(pp[2 * i]),
                                                          __int_as_float(pp[2 * i + 1]));
            ++round;
            __syncthreads();
        }
    }
    if (t == 0) {
        info[0] = round;
        info[1] = sweep;
        info[2] = converged;
    }
}

// ---------------------------------------------------------------- one-CTA Jacobi on the full matrix
// The same rotations in the same order as k_jacobi32 on the full s x s matrix
// (no index of a pair needs sorting) in place.  A round: thread k < np computes
// the rotation of pair k, while every thread loads its (at most IT) 2x2 blocks
// of the pair grid; after a barrier the threads update their blocks; a second
// barrier ends the round.  A thread keeps its blocks' pair numbers i, j over all
// rounds, and round r pairs r - k with r + k (mod m - 1) and m - 1 with r: a
// warp's blocks run along a row (m is even, so the pairs' diagonal and
// off-diagonal entries have odd strides as well: no bank conflicts).  This is the
// circle method on reversed indices, so k_apply_circle reads the log.
// The round is bound by its chain of latencies, pivot entries -> rotation ->
// table -> update, about 400 clocks at s = 64, and beyond that by the one SM's
// shared-memory accesses, eight a block.  GB300, kernel alone, k_jacobi32, the
// cluster kernel and this one: s = 30 66, 74, 29 us; s = 64 166, 151, 85 us;
// s = 96 391, 254, 229 us; s = 112 513, 307, 347 us: hence kJacCtaMax.  (Every warp
// computing all rotations for itself, with two copies of the matrix and one
// barrier: s = 30 28, s = 64 107 us.)
constexpr int kJacCtaMax = 104;  // np^2 blocks: at most 3 a thread

size_t jacobi_cta_smem_bytes(int s) {
    const int m = jac_m(s);
    return (size_t)m * m * sizeof(float);
}

template <int IT>
__global__ void __launch_bounds__(kJacobiThreads, 1)
k_jacobi_cta(int s, const double *__restrict__ M, int ldm, float2 *__restrict__ log,
             int max_rounds, int *__restrict__ info) {
    extern __shared__ float A[];  // m x m; the padding index of an odd s has zero entries
    __shared__ float red[2][32][2];
    __shared__ float2 tab[kJacCtaMax / 2];  // c, s of the round's pairs
    const int m = jac_m(s), np = m / 2, m1 = m - 1;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = blockDim.x >> 5;
    for (int idx = t; idx < m * m; idx += blockDim.x) {
        const int x = idx / m, y = idx - x * m;
        float v = 0.0f;
        if (x < s && y < s) v = (float)(0.5 * (M[x + (size_t)y * ldm] + M[y + (size_t)x * ldm]));
        A[idx] = v;
    }
    // the thread's blocks (row pair, column pair)
    int bi[IT], bj[IT];
#pragma unroll
    for (int u = 0; u < IT; ++u) {
        const int b = t + u * blockDim.x;
        bi[u] = b < np * np ? b / np : 0;
        bj[u] = b < np * np ? b - bi[u] * np : 0;
    }
    // indices of pair k in round r
    auto top = [&](int k, int r) {
        const int v = r - k;
        return k == 0 ? m1 : (v < 0 ? v + m1 : v);
    };
    auto bot = [&](int k, int r) {
        const int v = r + k;
        return v >= m1 ? v - m1 : v;
    };
    __syncthreads();
    int round = 0, sweep = 0, converged = 0;
    for (sweep = 0; sweep < kMaxSweeps && round + m1 <= max_rounds; ++sweep) {
        // stop when the off-diagonal mass is at the FP32 noise level
        float off = 0.0f, tot = 0.0f;
        for (int x = warp; x < m; x += nwarps)
            for (int y = lane; y < m; y += 32) {
                const float v = A[x * m + y] * A[x * m + y];
                tot += v;
                if (x != y) off += v;
            }
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if (lane == 0) {
            red[sweep & 1][warp][0] = off;
            red[sweep & 1][warp][1] = tot;
        }
        __syncthreads();
        off = tot = 0.0f;
        for (int w = 0; w < nwarps; ++w) {
            off += red[sweep & 1][w][0];
            tot += red[sweep & 1][w][1];
        }
        if (off <= kOffTol * kOffTol * tot) {  // the same sums in every thread
            converged = 1;
            break;
        }
        for (int r = 0; r < m1; ++r) {
            if (t < np) {
                const int p = top(t, r), q = bot(t, r);
                const float app = A[p * m + p], aqq = A[q * m + q], apq = A[p * m + q];
                float c = 1.0f, sv = 0.0f;
                const float thr = kRotTol * sqrtf(fabsf(app) * fabsf(aqq));
                if (fabsf(apq) > thr && fabsf(apq) > 1e-30f) {
                    // (an infinite tau^2 gives the rotation 0, as it should; tau = 0
                    // turns towards the larger index whichever of p, q that is)
                    const float tau = (aqq - app) / (2.0f * apq);
                    const float tt = ((p < q ? tau >= 0.0f : tau > 0.0f) ? 1.0f : -1.0f) /
                                     (fabsf(tau) + sqrtf(fmaf(tau, tau, 1.0f)));
                    c = rsqrtf(1.0f + tt * tt);
                    sv = tt * c;
                }
                tab[t] = make_float2(c, sv);
                log[(size_t)round * np + t] = make_float2(c, sv);
            }
            float d[IT][4];
#pragma unroll
            for (int u = 0; u < IT; ++u) {
                const float *rt = A + top(bi[u], r) * m, *rb = A + bot(bi[u], r) * m;
                const int p = top(bj[u], r), q = bot(bj[u], r);
                d[u][0] = rt[p];
                d[u][1] = rt[q];
                d[u][2] = rb[p];
                d[u][3] = rb[q];
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < IT; ++u) {
                if (t + u * (int)blockDim.x >= np * np) break;
                const float2 ei = tab[bi[u]], ej = tab[bj[u]];
                const float t11 = ei.x * d[u][0] - ei.y * d[u][2];
                const float t12 = ei.x * d[u][1] - ei.y * d[u][3];
                const float t21 = ei.y * d[u][0] + ei.x * d[u][2];
                const float t22 = ei.y * d[u][1] + ei.x * d[u][3];
                float *rt = A + top(bi[u], r) * m, *rb = A + bot(bi[u], r) * m;
                const int p = top(bj[u], r), q = bot(bj[u], r);
                const bool zero = bi[u] == bj[u] && ei.y != 0.0f;
                rt[p] = t11 * ej.x - t12 * ej.y;
                rt[q] = zero ? 0.0f : t11 * ej.y + t12 * ej.x;
                rb[p] = zero ? 0.0f : t21 * ej.x - t22 * ej.y;
                rb[q] = t21 * ej.y + t22 * ej.x;
            }
            __syncthreads();
            ++round;
        }
    }
    if (t == 0) {
        info[0] = round;
        info[1] = sweep;
        info[2] = converged;
    }
}

template <int IT>
static void launch_jacobi_cta(int s, const double *M, int ldm, float2 *log, int max_rounds,
                              int *info, cudaStream_t st) {
    static PerDevice<bool> smem_set;  // allow the largest size once per device
    smem_set.get([] {
        GCGE_CUDA(cudaFuncSetAttribute(k_jacobi_cta<IT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)jacobi_cta_smem_bytes(kJacCtaMax)));
        return true;
    });
    const int np = jac_m(s) / 2, threads = std::min(kJacobiThreads, (np * np + 31) / 32 * 32);
    k_jacobi_cta<IT><<<1, threads, jacobi_cta_smem_bytes(s), st>>>(s, M, ldm, log, max_rounds,
                                                                  info);
    GCGE_CHECK_LAUNCH();
}

// ---------------------------------------------------------------- cluster Jacobi
// The same rotations in a cluster of kJC CTAs.  Indices are arranged by the
// circle method: with P_r[0] = 0 and P_r[i] = 1 + ((i - 1 - r) mod (m - 1)),
// pair slot k of round r is (P_r[k], P_r[m - 1 - k]); after m - 1 rounds P is
// the identity again.  CTA c owns the slots [c np / kJC, (c + 1) np / kJC) and
// holds the two full rows (m floats each) of each of its slots.  A round:
//   (a) every CTA computes the rotations of its slots and writes them into the
//       round table of every CTA of the cluster;
//   (b) after a cluster barrier, each CTA updates every 2x2 block (own slot i,
//       any slot j) of its rows, A <- J^T A J, and writes the new rows into
//       the other row buffer at the slots they hold in the next round, which
//       for at most two rows per CTA is in the neighbouring CTA's shared
//       memory;
//   (c) a second cluster barrier makes the next buffers complete.
// The round is bound by the latency of its serial chain.  A form with one
// barrier, in which every CTA computed all rotations from a table of the pairs'
// entries that the block updates of the previous round kept up to date, paid
// more in the updates than the barrier costs (kernel, one barrier against two:
// s = 105 978 and 1043 us, 128 1512 and 1451, 180 2452 and 2404, 260 5857 and
// 4325, 460 17.3 and 13.8 ms).
// The stopping test is that of k_jacobi32; every CTA sums the per-CTA
// off-diagonal masses in the same order, so all take the same decision.
constexpr int kJC = 8;
constexpr int kJacMaxLocal = 32;    // slots per CTA (np <= 256: s <= 512)

__host__ __device__ inline int jc_slots(int np) { return (np + kJC - 1) / kJC; }

size_t jacobi_cluster_smem_bytes(int s) {
    const int m = jac_m(s), np = m / 2, ks = jc_slots(np);
    return (size_t)np * sizeof(float4) + (size_t)2 * 2 * ks * m * sizeof(float) +
           (size_t)2 * kJC * 2 * sizeof(float) + 64;
}

// index at position i < m1 + 1 of the circle arrangement after r < m1 rounds
__device__ __forceinline__ int circle_index(int i, int r, int m1) {
    if (i == 0) return 0;
    const int v = i - 1 - r;
    return 1 + (v < 0 ? v + m1 : v);
}

// CTA owning slot k (slots [c np / kJC, (c + 1) np / kJC) belong to CTA c)
__device__ __forceinline__ int slot_owner(int k, int np) { return ((k + 1) * kJC - 1) / np; }

__global__ void __launch_bounds__(kJacobiThreads, 1)
k_jacobi32_cluster(int s, const double *__restrict__ M, int ldm, float2 *__restrict__ log,
                   int max_rounds, int *__restrict__ info) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    extern __shared__ __align__(16) unsigned char jsm[];
    const int m = jac_m(s), np = m / 2, ks = jc_slots(np), m1 = m - 1;
    float4 *tab = reinterpret_cast<float4 *>(jsm);          // [np]: c, s, p, q of the round
    float *rows = reinterpret_cast<float *>(tab + np);      // [2][2 ks][m]
    float *red = rows + (size_t)2 * 2 * ks * m;               // [2][kJC][2]
    __shared__ float wsum[kJacobiThreads / 32][2];
    __shared__ int stop;
    __shared__ float *s_dst[2 * kJacMaxLocal];  // next-round places of the local rows
    const size_t bufsz = (size_t)2 * ks * m;
    const int k0 = (rank * np) / kJC, k1 = ((rank + 1) * np) / kJC, nloc = k1 - k0;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = blockDim.x >> 5;
    // rows of round 0 (P = identity): slot k holds rows k and m - 1 - k
    for (int idx = t; idx < 2 * nloc * m; idx += blockDim.x) {
        const int lr = idx / m, y = idx - lr * m;
        const int k = k0 + (lr >> 1);
        const int x = (lr & 1) ? m - 1 - k : k;
        float v = 0.0f;
        if (x < s && y < s) v = (float)(0.5 * (M[x + (size_t)y * ldm] + M[y + (size_t)x * ldm]));
        rows[(size_t)lr * m + y] = v;
    }
    cl.sync();  // every CTA of the cluster runs before any remote access
    int cur = 0, round = 0, sweep = 0, converged = 0;
    for (sweep = 0; sweep < kMaxSweeps && round + m1 <= max_rounds; ++sweep) {
        // off-diagonal mass at the start of the sweep (P = identity again)
        {
            const float *R = rows + cur * bufsz;
            float off = 0.0f, tot = 0.0f;
            for (int idx = t; idx < 2 * nloc * m; idx += blockDim.x) {
                const int lr = idx / m, y = idx - lr * m;
                const int k = k0 + (lr >> 1);
                const int x = (lr & 1) ? m - 1 - k : k;
                const float v = R[(size_t)lr * m + y];
                tot += v * v;
                if (x != y) off += v * v;
            }
            for (int o = 16; o > 0; o >>= 1) {
                off += __shfl_xor_sync(0xffffffffu, off, o);
                tot += __shfl_xor_sync(0xffffffffu, tot, o);
            }
            if (lane == 0) {
                wsum[warp][0] = off;
                wsum[warp][1] = tot;
            }
            __syncthreads();
            if (t == 0) {
                float a = 0.0f, b = 0.0f;
                for (int w = 0; w < nwarps; ++w) {
                    a += wsum[w][0];
                    b += wsum[w][1];
                }
                float *slot = red + ((sweep & 1) * kJC + rank) * 2;
                for (int c = 0; c < kJC; ++c) {
                    float *dst = cl.map_shared_rank(slot, c);
                    dst[0] = a;
                    dst[1] = b;
                }
            }
            cl.sync();
            if (t == 0) {
                float a = 0.0f, b = 0.0f;
                for (int c = 0; c < kJC; ++c) {
                    a += red[((sweep & 1) * kJC + c) * 2];
                    b += red[((sweep & 1) * kJC + c) * 2 + 1];
                }
                stop = (a <= kOffTol * kOffTol * b) ? 1 : 0;
            }
            __syncthreads();
            if (stop) {
                converged = 1;
                break;
            }
        }
        for (int r = 0; r < m1; ++r) {
            const float *R = rows + cur * bufsz;
            // (a) the rotations of the local slots, into every CTA's table
            for (int k = k0 + t; k < k1; k += blockDim.x) {
                const int p = circle_index(k, r, m1), q = circle_index(m - 1 - k, r, m1);
                float c = 1.0f, sv = 0.0f;
                if (p < s && q < s) {
                    const float *top = R + (size_t)(2 * (k - k0)) * m;
                    const float app = top[p], aqq = top[m + q], apq = top[q];
                    const float thr = kRotTol * sqrtf(fabsf(app) * fabsf(aqq));
                    if (fabsf(apq) > thr && fabsf(apq) > 1e-30f) {
                        // (an infinite tau^2 gives the rotation 0, as it should)
                        const float tau = (aqq - app) / (2.0f * apq);
                        const float tt = (tau >= 0.0f ? 1.0f : -1.0f) /
                                         (fabsf(tau) + sqrtf(fmaf(tau, tau, 1.0f)));
                        c = rsqrtf(1.0f + tt * tt);
                        sv = tt * c;
                    }
                }
                const float4 e = make_float4(c, sv, __int_as_float(p), __int_as_float(q));
#pragma unroll
                for (int o = 0; o < kJC; ++o) *cl.map_shared_rank(tab + k, o) = e;
                log[(size_t)round * np + k] = make_float2(c, sv);
            }
            // next-round places of the local rows (circle method)
            for (int lr = (int)blockDim.x - 1 - t; lr < 2 * nloc; lr += blockDim.x) {
                const int k = k0 + (lr >> 1);
                int kn, sn;
                if (np == 1) kn = 0, sn = lr & 1;
                else if (lr & 1) kn = k == 0 ? 1 : k - 1, sn = k == 0 ? 0 : 1;
                else if (k == 0) kn = 0, sn = 0;
                else if (k <= np - 2) kn = k + 1, sn = 0;
                else kn = np - 1, sn = 1;
                const int o = slot_owner(kn, np);
                float *d = rows + (size_t)(cur ^ 1) * bufsz +
                           (size_t)(2 * (kn - (o * np) / kJC) + sn) * m;
                s_dst[lr] = o == rank ? d : cl.map_shared_rank(d, o);
            }
            cl.sync();
            // (b) the 2x2 blocks of the local rows, written to the next buffers
            const float inv_np = 1.0f / (float)np;  // b / np exactly: the quotient's
#pragma unroll 2
            for (int b = t; b < nloc * np; b += blockDim.x) {  // fraction is >= 0.5 / np away
                const int li = (int)(((float)b + 0.5f) * inv_np);
                const int j = b - li * np;
                const int ki = k0 + li;
                const float4 ei = tab[ki], ej = tab[j];
                const float ci = ei.x, si = ei.y, cj = ej.x, sj = ej.y;
                const int pj = __float_as_int(ej.z), qj = __float_as_int(ej.w);
                const float *Tp = R + (size_t)(2 * li) * m, *Tq = Tp + m;
                float o11, o12, o21, o22;
                if (ki == j) {
                    const float app = Tp[pj], aqq = Tq[qj], apq = Tp[qj], aqp = Tq[pj];
                    if (si != 0.0f) {
                        const float t11 = ci * app - si * apq, t12 = ci * apq - si * aqq;
                        const float t21 = si * app + ci * apq, t22 = si * apq + ci * aqq;
                        o11 = t11 * ci - t12 * si;
                        o22 = t21 * si + t22 * ci;
                        o12 = o21 = 0.0f;
                    } else {
                        o11 = app;
                        o12 = apq;
                        o21 = aqp;
                        o22 = aqq;
                    }
                } else {
                    const float a11 = Tp[pj], a12 = Tp[qj], a21 = Tq[pj], a22 = Tq[qj];
                    const float t11 = ci * a11 - si * a21, t12 = ci * a12 - si * a22;
                    const float t21 = si * a11 + ci * a21, t22 = si * a12 + ci * a22;
                    o11 = t11 * cj - t12 * sj;
                    o12 = t11 * sj + t12 * cj;
                    o21 = t21 * cj - t22 * sj;
                    o22 = t21 * sj + t22 * cj;
                }
                float *dt = s_dst[2 * li], *db = s_dst[2 * li + 1];
                dt[pj] = o11;
                dt[qj] = o12;
                db[pj] = o21;
                db[qj] = o22;
            }
            cl.sync();
            cur ^= 1;
            ++round;
        }
    }
    if (rank == 0 && t == 0) {
        info[0] = round;
        info[1] = sweep;
        info[2] = converged;
    }
    cl.sync();  // no CTA leaves while another may still address its memory
}

// Largest dynamic shared memory the Jacobi kernel may request: the device's
// opt-in per-block limit minus the kernel's static shared memory.
static size_t jacobi_dyn_limit() {
    static PerDevice<size_t> cache;
    return cache.get([] {
        int optin = 0;
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, current_device());
        cudaFuncAttributes fa{};
        cudaFuncGetAttributes(&fa, k_jacobi32);
        return optin > 0 ? (size_t)optin - fa.sharedSizeBytes : (size_t)48 * 1024;
    });
}
// the same for the cluster kernel (its static shared memory differs)
static size_t jacobi_cluster_dyn_limit() {
    static PerDevice<size_t> cache;
    return cache.get([] {
        int optin = 0;
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, current_device());
        cudaFuncAttributes fa{};
        cudaFuncGetAttributes(&fa, k_jacobi32_cluster);
        return optin > 0 ? (size_t)optin - fa.sharedSizeBytes : (size_t)48 * 1024;
    });
}

// V = J_1 J_2 ... J_T, one warp per row of V: row r starts as e_r and every
// logged rotation (c, s, p, q) maps (v_p, v_q) -> (c v_p - s v_q, s v_p + c v_q).
// Lane l applies the rotations of pairs l, l + 32, ... (NS slots); the log of
// the next kRotGroup rounds is loaded while the current ones are applied, so
// the row's updates do not wait on the log's L2 latency.
constexpr int kRotGroup = 2;
template <int NS>
__global__ void __launch_bounds__(256)
k_apply_rotations(int s, const float4 *__restrict__ log, const int *__restrict__ info,
                  double *__restrict__ V, int ldv) {
    extern __shared__ float rows[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 8 + warp;
    if (r >= s) return;  // warp-uniform; the kernel has no block-wide barrier
    float *v = rows + (size_t)warp * s;
    const int np = jac_m(s) / 2;
    const int rounds = info[0];
    for (int j = lane; j < s; j += 32) v[j] = (j == r) ? 1.0f : 0.0f;
    __syncwarp();
    auto load = [&](float4 (&dst)[kRotGroup][NS], int t0) {
#pragma unroll
        for (int g = 0; g < kRotGroup; ++g)
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                const int i = lane + 32 * k;
                dst[g][k] = (t0 + g < rounds && i < np) ? log[(size_t)(t0 + g) * np + i]
                                                        : make_float4(1.0f, 0.0f, 0.0f, 0.0f);
            }
    };
    float4 cur[kRotGroup][NS], nxt[kRotGroup][NS];
    load(cur, 0);
    for (int t0 = 0; t0 < rounds; t0 += kRotGroup) {
        load(nxt, t0 + kRotGroup);
#pragma unroll
        for (int g = 0; g < kRotGroup; ++g) {
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                const float4 e = cur[g][k];
                if (e.y == 0.0f) continue;  // also every slot past np or past the last round
                const int p = __float_as_int(e.z), q = __float_as_int(e.w);
                if (p >= s || q >= s) continue;
                const float vp = v[p], vq = v[q];
                v[p] = e.x * vp - e.y * vq;
                v[q] = e.y * vp + e.x * vq;
            }
            __syncwarp();
        }
#pragma unroll
        for (int g = 0; g < kRotGroup; ++g)
#pragma unroll
            for (int k = 0; k < NS; ++k) cur[g][k] = nxt[g][k];
    }
    for (int j = lane; j < s; j += 32) V[r + (size_t)j * ldv] = (double)v[j];
}

template <int NS>
static void launch_rotations(int s, const float4 *log, const int *info, double *V, int ldv,
                             cudaStream_t st) {
    k_apply_rotations<NS><<<(s + 7) / 8, 256, (size_t)8 * s * sizeof(float), st>>>(s, log, info,
                                                                                  V, ldv);
}

// The same product from the cluster kernel's log, whose rounds follow the
// circle method: slot k's pair sits at positions k and m - 1 - k of the
// arrangement, and between rounds every entry moves on by one position.  A
// warp holds its row by position in registers (lane l slots [l NS, (l + 1) NS):
// the two entries of each), rotates the slots' pairs and moves the entries, one
// of each end to the neighbouring lanes, so that a round is a dozen dependent
// instructions and no memory but the log (c, s per slot), which the kernel
// reads kCircleAhead rounds ahead.  The arrangement is back at the identity
// after whole sweeps, which is all that the log holds.  s = 180: 92 us through
// shared memory, with the pairs' indices read from the log.
constexpr int kCircleAhead = 4;
template <int NS>
__global__ void __launch_bounds__(128)
k_apply_circle(int s, const float2 *__restrict__ log, const int *__restrict__ info,
               double *__restrict__ V, int ldv, bool reversed) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * 4 + warp;
    if (row >= s) return;  // warp-uniform; the kernel has no block-wide barrier
    const int m = jac_m(s), np = m / 2, rounds = info[0];
    const int k0 = lane * NS, pos = reversed ? m - 1 - row : row;
    float top[NS], bot[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        top[j] = k0 + j == pos ? 1.0f : 0.0f;
        bot[j] = m - 1 - (k0 + j) == pos ? 1.0f : 0.0f;
    }
    float2 q[kCircleAhead][NS];
    auto load = [&](float2 (&dst)[NS], int t) {
#pragma unroll
        for (int j = 0; j < NS; ++j)
            dst[j] = (t < rounds && k0 + j < np) ? __ldg(log + (size_t)t * np + k0 + j)
                                                 : make_float2(1.0f, 0.0f);
    };
    auto step = [&](const float2 (&e)[NS]) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            const float vt = top[j], vb = bot[j];
            top[j] = e[j].x * vt - e[j].y * vb;
            bot[j] = e[j].y * vt + e[j].x * vb;
        }
        if (NS == 1 && np == 1) return;  // a single pair stays where it is
        // top k -> top k + 1, bottom k -> bottom k - 1; top 0 stays, bottom 0 ->
        // top 1, top np - 1 -> bottom np - 1
        const float b0 = bot[0];
        const float from_left = __shfl_up_sync(0xffffffffu, NS == 1 && lane == 0 ? b0 : top[NS - 1], 1);
        const float from_right = __shfl_down_sync(0xffffffffu, b0, 1);
        const float first = top[0];
        float nt[NS], nb[NS];
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            nt[j] = j == 0 ? from_left : (j == 1 && lane == 0 ? b0 : top[j - 1]);
            nb[j] = k0 + j == np - 1 ? top[j] : (j + 1 < NS ? bot[j + 1 < NS ? j + 1 : j] : from_right);
        }
        if (lane == 0) nt[0] = first;
#pragma unroll
        for (int j = 0; j < NS; ++j) top[j] = nt[j], bot[j] = nb[j];
    };
#pragma unroll
    for (int g = 0; g < kCircleAhead; ++g) load(q[g], g);
    for (int t0 = 0; t0 < rounds; t0 += kCircleAhead) {
#pragma unroll
        for (int g = 0; g < kCircleAhead; ++g) {
            if (t0 + g < rounds) step(q[g]);  // warp-uniform
            load(q[g], t0 + g + kCircleAhead);
        }
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        const int k = k0 + j, ct = reversed ? m - 1 - k : k, cb = m - 1 - ct;
        if (k < np) {
            if (ct < s) V[row + (size_t)ct * ldv] = (double)top[j];
            if (cb < s) V[row + (size_t)cb * ldv] = (double)bot[j];
        }
    }
}

// Whether a cluster of kJC CTAs with the largest shared memory the cluster
// kernel may use can be resident on this device (checked once).
static bool jacobi_cluster_usable() {
    static PerDevice<bool> cache;
    return cache.get([] {
        const size_t lim = jacobi_cluster_dyn_limit();
        if (cudaFuncSetAttribute(k_jacobi32_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)lim) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kJC);
        cfg.blockDim = dim3(kJacobiThreads);
        cfg.dynamicSmemBytes = lim;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kJC;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_jacobi32_cluster, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return n > 0;
    });
}

static int jacobi_cluster_max_dim() {
    const size_t lim = jacobi_cluster_dyn_limit();
    int s = kJacCtaMax;
    while (jacobi_cluster_smem_bytes(s + 1) <= lim && jc_slots(jac_m(s + 1) / 2) <= kJacMaxLocal)
        ++s;
    return s;
}

void EigWork::reserve(int smax) {
    const size_t s2 = (size_t)smax * smax;
    G.alloc(s2);
    W.alloc(s2);
    S.alloc(s2);
    C.alloc(s2);
    X.alloc(s2);
    X2.alloc(s2);
    lam.alloc(smax);
    delta.alloc(4);
    info.alloc(4);
    const int m = jac_m(smax);
    max_rounds = kMaxSweeps * (m - 1);
    log.alloc((size_t)max_rounds * (m / 2) + 1);  // (c, s, p, q) per pair and round
    gscr.alloc(gram_scratch_elems(smax, smax, smax));
    ozb.alloc(oz_lincomb_scratch_bytes(smax, smax));
    h_S.alloc(s2);
    h_C.alloc(2 * s2);
    h_lam.alloc(smax);
    h_info.alloc(8);
    std::fill(h_info.p, h_info.p + 8, 0.0);
    cap = smax;
}

// Cyclic FP64 Jacobi on a small dense symmetric block (host, row-major n x n
// in a), eigenvectors accumulated in v (column j = eigenvector j).
static void host_jacobi(int n, std::vector<double> &a, std::vector<double> &v) {
    v.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; ++i) v[(size_t)i * n + i] = 1.0;
    for (int sweep = 0; sweep < 60; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) {
                tot += a[(size_t)i * n + j] * a[(size_t)i * n + j];
                if (i != j) off += a[(size_t)i * n + j] * a[(size_t)i * n + j];
            }
        if (off <= 1e-34 * tot || off == 0.0) break;
        for (int p = 0; p < n - 1; ++p)
            for (int q = p + 1; q < n; ++q) {
                const double apq = a[(size_t)p * n + q];
                if (apq == 0.0) continue;
                const double app = a[(size_t)p * n + p], aqq = a[(size_t)q * n + q];
                const double tau = (aqq - app) / (2.0 * apq);
                const double tt = (tau >= 0 ? 1.0 : -1.0) / (std::fabs(tau) + std::hypot(1.0, tau));
                const double c = 1.0 / std::sqrt(1.0 + tt * tt), sv = tt * c;
                for (int k = 0; k < n; ++k) {  // A <- A J (columns p, q)
                    const double akp = a[(size_t)k * n + p], akq = a[(size_t)k * n + q];
                    a[(size_t)k * n + p] = c * akp - sv * akq;
                    a[(size_t)k * n + q] = sv * akp + c * akq;
                }
                for (int k = 0; k < n; ++k) {  // A <- J^T A (rows p, q)
                    const double apk = a[(size_t)p * n + k], aqk = a[(size_t)q * n + k];
                    a[(size_t)p * n + k] = c * apk - sv * aqk;
                    a[(size_t)q * n + k] = sv * apk + c * aqk;
                }
                for (int k = 0; k < n; ++k) {
                    const double vkp = v[(size_t)k * n + p], vkq = v[(size_t)k * n + q];
                    v[(size_t)k * n + p] = c * vkp - sv * vkq;
                    v[(size_t)k * n + q] = sv * vkp + c * vkq;
                }
            }
    }
}

void host_eigh(int n, const double *G, double *w, double *V) {
    std::vector<double> a(G, G + (size_t)n * n), v;
    for (int i = 0; i < n; ++i)  // symmetrise (column-major in, row-major work)
        for (int j = 0; j < i; ++j) {
            const double m = 0.5 * (a[(size_t)i * n + j] + a[(size_t)j * n + i]);
            a[(size_t)i * n + j] = a[(size_t)j * n + i] = m;
        }
    host_jacobi(n, a, v);
    std::vector<int> ord(n);
    for (int i = 0; i < n; ++i) ord[i] = i;
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) {
        return a[(size_t)x * n + x] < a[(size_t)y * n + y];
    });
    for (int j = 0; j < n; ++j) {
        w[j] = a[(size_t)ord[j] * n + ord[j]];
        for (int i = 0; i < n; ++i) V[i + (size_t)j * n] = v[(size_t)i * n + ord[j]];
    }
}

// Eigen-decomposition of the symmetric s x s matrix M (device, ld) into
// ascending eigenvalues eval (host) and eigenvectors Z (device, ldz).
//
// Refinement step (after Ogita & Aishima): with G = X^T X, R = I - G and
// S = X^T M X, lambda_i = S_ii / G_ii and X <- X (I + E), where
// E_ij = (S_ij + lambda_j R_ij) / (lambda_j - lambda_i) for well-separated
// pairs and R_ij / 2 inside a cluster.  A cluster is a connected set of
// pairs whose first-order correction is not small (|E_ij| > 1e-2) or whose
// gap is below 1e-5 max|lambda| (there E_ij would mostly amplify rounding);
// each cluster block of S is diagonalised exactly in FP64 in the same step,
// so near-degenerate pairs come out orthonormal and resolved to FP64
// accuracy.  The update of a step with max|E| < 1e-9 is the last (its error
// is of the order max|E|^2 / gap); that step folds the ascending sort into the
// update and writes Z.
int sym_eig(EigWork &wk, int s, const double *M, int ld, double *eval_host, double *Z, int ldz,
            int refine_steps, cudaStream_t st, bool emulated) {
    GCGE_REQUIRE(s >= 1 && s <= wk.cap, GCGE_ERR_ARG, "sym_eig: size");
    {  // counts of the previous call (its copy has completed by now: every
       // caller synchronises the stream between two eigensolves)
        const int *hi = reinterpret_cast<const int *>(wk.h_info.p);
        wk.last_rounds = hi[0];
        wk.last_sweeps = hi[1];
    }
    GCGE_REQUIRE(s <= jacobi_max_dim(), GCGE_ERR_TOO_LARGE,
                 "sym_eig: projected dimension exceeds the shared-memory Jacobi capacity");
    static PerDevice<bool> smem_set;  // allow the largest size once per device
    smem_set.get([] {
        GCGE_CUDA(cudaFuncSetAttribute(k_jacobi32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)jacobi_dyn_limit()));
        return true;
    });
    const bool cta = s <= kJacCtaMax;
    const bool cluster = !cta && jacobi_cluster_usable() &&
                         jacobi_cluster_smem_bytes(s) <= jacobi_cluster_dyn_limit() &&
                         jc_slots(jac_m(s) / 2) <= kJacMaxLocal;
    if (cluster || cta) {
        float2 *log = reinterpret_cast<float2 *>(wk.log.p);
        if (cta) {
            const int np = jac_m(s) / 2;
            auto go = np <= 32   ? launch_jacobi_cta<1>
                      : np <= 45 ? launch_jacobi_cta<2>
                                 : launch_jacobi_cta<3>;  // 52^2 = 2704 blocks
            go(s, M, ld, log, wk.max_rounds, wk.info.p, st);
        } else {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(kJC);
            cfg.blockDim = dim3(kJacobiThreads);
            cfg.dynamicSmemBytes = jacobi_cluster_smem_bytes(s);
            cfg.stream = st;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = kJC;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            GCGE_CUDA(cudaLaunchKernelEx(&cfg, k_jacobi32_cluster, s, M, ld, log, wk.max_rounds,
                                         wk.info.p));
            GCGE_CHECK_LAUNCH();
        }
        const int grid = (s + 3) / 4;
        switch ((jac_m(s) / 2 + 31) / 32) {
#define GCGE_CIRCLE_CASE(NS)                                                        \
    case NS:                                                                        \
        k_apply_circle<NS><<<grid, 128, 0, st>>>(s, log, wk.info.p, wk.X.p, s, cta); \
        break;
            GCGE_CIRCLE_CASE(1) GCGE_CIRCLE_CASE(2) GCGE_CIRCLE_CASE(3) GCGE_CIRCLE_CASE(4)
            GCGE_CIRCLE_CASE(5) GCGE_CIRCLE_CASE(6) GCGE_CIRCLE_CASE(7) GCGE_CIRCLE_CASE(8)
#undef GCGE_CIRCLE_CASE
            default: throw CudaError{GCGE_ERR_TOO_LARGE, "sym_eig: size"};
        }
    } else {
        GCGE_REQUIRE(jacobi_smem_bytes(s) <= jacobi_dyn_limit(), GCGE_ERR_TOO_LARGE,
                     "sym_eig: projected dimension exceeds the one-CTA Jacobi capacity");
        k_jacobi32<<<1, kJacobiThreads, jacobi_smem_bytes(s), st>>>(s, M, ld, wk.log.p,
                                                                    wk.max_rounds, wk.info.p);
        GCGE_CHECK_LAUNCH();
        switch ((jac_m(s) / 2 + 31) / 32) {
            case 2: launch_rotations<2>(s, wk.log.p, wk.info.p, wk.X.p, s, st); break;
            case 3: launch_rotations<3>(s, wk.log.p, wk.info.p, wk.X.p, s, st); break;
            case 4: launch_rotations<4>(s, wk.log.p, wk.info.p, wk.X.p, s, st); break;
            case 5: launch_rotations<5>(s, wk.log.p, wk.info.p, wk.X.p, s, st); break;
            default: launch_rotations<6>(s, wk.log.p, wk.info.p, wk.X.p, s, st); break;
        }
    }
    GCGE_CHECK_LAUNCH();
    count_launch(2);
    const int lds = s;
    double *X = wk.X.p, *Xn = wk.X2.p;
    // s x s products of the refinement: X^T P (ld s) and A B (ld of A given), on
    // the digit kernels from the size where these are faster than the FP64 units
    // (GB300, digits against FP64: X^T P 37 against 16 us at s = 180, 42 against
    // 113 at 400; A B 51 against 16 and 81 against 113).  Largest error of an entry
    // over |x||p| at s = 180, FP64 and digits: 2.5e-16 and 0.7e-16 for orthogonal
    // columns, 3.2e-16 and 2.2e-16 with 8 decades of row scales: either is FP64
    // rounding, as in the FP64 solve, and the next step corrects it
    const double flops = 2.0 * s * s * s;
    const bool digit_gram = emulated && flops > 2.8e7, digit_lincomb = emulated && flops > 6e7;
    auto sgram = [&](const double *P, double *C) {
        if (digit_gram)
            oz_gram(s, s, s, X, lds, P, lds, C, lds, wk.gscr.p, wk.gscr.n, st);
        else
            gram(s, s, s, X, lds, P, lds, C, lds, wk.gscr.p, wk.gscr.n, st);
    };
    auto slincomb = [&](const double *A, int lda, const double *B, double *Y, int ldy) {
        if (digit_lincomb)
            oz_lincomb(s, s, s, A, lda, B, lds, Y, ldy, nullptr, 0, st, 1.0, wk.ozb.p, wk.ozb.n);
        else
            lincomb(s, s, s, A, lda, B, lds, Y, ldy, nullptr, 0, st);
    };
    const size_t s2 = (size_t)s * s;
    double *hS = wk.h_S.p, *hG = wk.h_C.p + s2, *hC = wk.h_C.p;
    std::vector<double> lam(s);
    std::vector<int> ord(s), comp(s), parent(s);
    auto find = [&](int x) {
        while (parent[x] != x) {
            parent[x] = parent[parent[x]];
            x = parent[x];
        }
        return x;
    };
    const int steps = std::max(2, refine_steps);
    for (int step = 0; step < steps; ++step) {
        sgram(X, wk.G.p);
        slincomb(M, ld, X, wk.W.p, lds);
        sgram(wk.W.p, wk.S.p);
        GCGE_CUDA(cudaMemcpyAsync(hS, wk.S.p, sizeof(double) * s2, cudaMemcpyDeviceToHost, st));
        GCGE_CUDA(cudaMemcpyAsync(hG, wk.G.p, sizeof(double) * s2, cudaMemcpyDeviceToHost, st));
        GCGE_CUDA(cudaStreamSynchronize(st));
        double scale = 0.0;
        for (int i = 0; i < s; ++i) {
            lam[i] = hS[i + (size_t)i * s] / hG[i + (size_t)i * s];
            GCGE_REQUIRE(std::isfinite(lam[i]), GCGE_ERR_NUMERIC, "sym_eig: non-finite eigenvalue");
            scale = std::max(scale, std::fabs(lam[i]));
        }
        // E_ij = (S_ij + lam_j R_ij) / (lam_j - lam_i); pairs whose correction is
        // not small, or whose gap is below kClusterGap * scale, join one cluster
        for (int i = 0; i < s; ++i) parent[i] = i;
        for (int j = 0; j < s; ++j)
            for (int i = 0; i < s; ++i) {
                const double rij = (i == j ? 1.0 : 0.0) - hG[i + (size_t)j * s];
                double e = 0.5 * rij;
                if (i != j) {
                    const double gap = lam[j] - lam[i];
                    e = (hS[i + (size_t)j * s] + lam[j] * rij) / gap;
                    if (!(std::fabs(gap) > kClusterGap * scale) || !(std::fabs(e) <= kStrongCoupling)) {
                        const int a = find(i), b = find(j);
                        if (a != b) parent[a] = b;
                    }
                }
                hC[i + (size_t)j * s] = e;  // E for now
            }
        for (int i = 0; i < s; ++i) comp[i] = find(i);
        double emax = 0.0;
        for (int j = 0; j < s; ++j)
            for (int i = 0; i < s; ++i) {
                double &e = hC[i + (size_t)j * s];
                if (i != j && comp[i] == comp[j]) e = 0.5 * ((i == j ? 1.0 : 0.0) - hG[i + (size_t)j * s]);
                emax = std::max(emax, std::fabs(e));
                if (i == j) e += 1.0;  // C = I + E
            }
        // exact FP64 diagonalisation of each cluster block of S
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) {
            return comp[a] != comp[b] ? comp[a] < comp[b] : a < b;
        });
        int k = 0;
        while (k < s) {
            int e = k + 1;
            while (e < s && comp[ord[e]] == comp[ord[k]]) ++e;
            const int c = e - k;
            if (c > 1) {
                // the cluster block of (I + E)^T S (I + E): its in-cluster part
                // T = I + E_c (first-order G_c^{-1/2}) carries the off-diagonal
                // Gram entries, so the block's eigenvalues are accurate to
                // second order in them; the cross terms through entries of E
                // outside the cluster are second order too
                std::vector<double> Sc((size_t)c * c), Tc((size_t)c * c), ST((size_t)c * c);
                std::vector<double> blk((size_t)c * c), vec;
                for (int a = 0; a < c; ++a)
                    for (int b = 0; b < c; ++b) {
                        const int ia = ord[k + a], ib = ord[k + b];
                        Sc[(size_t)a * c + b] = 0.5 * (hS[ia + (size_t)ib * s] + hS[ib + (size_t)ia * s]);
                        Tc[(size_t)a * c + b] = hC[ia + (size_t)ib * s];  // row a, column b
                    }
                for (int a = 0; a < c; ++a)  // ST = Sc Tc
                    for (int b = 0; b < c; ++b) {
                        double v = 0.0;
                        for (int u = 0; u < c; ++u) v += Sc[(size_t)a * c + u] * Tc[(size_t)u * c + b];
                        ST[(size_t)a * c + b] = v;
                    }
                for (int a = 0; a < c; ++a)  // blk = Tc^T ST
                    for (int b = 0; b < c; ++b) {
                        double v = 0.0;
                        for (int u = 0; u < c; ++u) v += Tc[(size_t)u * c + a] * ST[(size_t)u * c + b];
                        blk[(size_t)a * c + b] = v;
                    }
                for (int a = 0; a < c; ++a)
                    for (int b = 0; b < a; ++b) {
                        const double v = 0.5 * (blk[(size_t)a * c + b] + blk[(size_t)b * c + a]);
                        blk[(size_t)a * c + b] = blk[(size_t)b * c + a] = v;
                    }
                host_jacobi(c, blk, vec);
                std::vector<double> tmp((size_t)s * c, 0.0);
                for (int b = 0; b < c; ++b)
                    for (int a = 0; a < c; ++a) {
                        const double v = vec[(size_t)a * c + b];
                        if (v == 0.0) continue;
                        const double *src = hC + (size_t)ord[k + a] * s;
                        double *dst = tmp.data() + (size_t)b * s;
                        for (int i = 0; i < s; ++i) dst[i] += src[i] * v;
                    }
                for (int b = 0; b < c; ++b) {
                    std::copy(tmp.begin() + (size_t)b * s, tmp.begin() + (size_t)(b + 1) * s,
                              hC + (size_t)ord[k + b] * s);
                    lam[ord[k + b]] = blk[(size_t)b * c + b];
                }
            }
            k = e;
        }
        // the step's error is second order in emax (first order inside clusters,
        // which are diagonalised exactly), so once emax < 1e-9 this update is
        // the last one needed
        const bool last = (step == steps - 1) || emax < 1e-9;
        wk.last_steps = step + 1;
        if (!last) {
            GCGE_CUDA(cudaMemcpyAsync(wk.C.p, hC, sizeof(double) * s2, cudaMemcpyHostToDevice, st));
            slincomb(X, lds, wk.C.p, Xn, lds);
            std::swap(X, Xn);
            // hC is rewritten only after the next step's synchronisation, which
            // follows this copy on the stream
            continue;
        }
        // final: ascending order folded into the update
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return lam[a] < lam[b]; });
        double *hP = wk.h_S.p;  // S is no longer needed
        for (int j = 0; j < s; ++j) {
            std::copy(hC + (size_t)ord[j] * s, hC + (size_t)(ord[j] + 1) * s, hP + (size_t)j * s);
            eval_host[j] = lam[ord[j]];
        }
        GCGE_CUDA(cudaMemcpyAsync(wk.C.p, hP, sizeof(double) * s2, cudaMemcpyHostToDevice, st));
        slincomb(X, lds, wk.C.p, Z, ldz);
        wk.last_delta = emax;
        break;
    }
    // the Jacobi's round and sweep counts reach the host with the caller's
    // next synchronisation (no wait here); the next call reads them
    GCGE_CUDA(cudaMemcpyAsync(wk.h_info.p, wk.info.p, sizeof(int) * 3, cudaMemcpyDeviceToHost,
                              st));
    return GCGE_OK;
}

}  // namespace gcge
