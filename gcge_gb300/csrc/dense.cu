// Dense multivector kernels (FP64 unless noted): axpby, the tall-skinny
// products X*C (MultiVecLinearComb, Ritz vectors, P) and Q^T P (inner products,
// Gram blocks of Rayleigh-Ritz and B-orthogonalisation), column dots and
// small helpers.
//
// FP64 on GB300 issues about two FMAs per clock per SM (measured 1.2 TFLOP/s
// for the whole part against 70 TFLOP/s FP32), so the products are FP64-FMA
// bound, not HBM bound: the kernels keep every SM busy (split-K for Q^T P,
// small tiles for small outputs) rather than chasing data reuse.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace gcge {

static int num_sms() { return device_sms(); }

// ---------------------------------------------------------------- axpby
template <typename T>
__global__ void k_axpby(int n, int ncols, T alpha, const T *__restrict__ X, int ldx, T beta,
                        T *__restrict__ Y, int ldy) {
    const size_t total = (size_t)n * ncols;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        T y = beta == T(0) ? T(0) : beta * Y[i + (size_t)c * ldy];
        if (X != nullptr && alpha != T(0)) y = fma(alpha, X[i + (size_t)c * ldx], y);
        Y[i + (size_t)c * ldy] = y;
    }
}

static int grid_for(size_t total, int threads) {
    size_t b = (total + threads - 1) / threads;
    size_t cap = (size_t)num_sms() * 16;
    return (int)std::max<size_t>(1, std::min(b, cap));
}

void axpby(int n, int ncols, double alpha, const double *X, int ldx, double beta, double *Y,
           int ldy, cudaStream_t st) {
    if (n <= 0 || ncols <= 0) return;
    k_axpby<double><<<grid_for((size_t)n * ncols, 256), 256, 0, st>>>(n, ncols, alpha, X, ldx,
                                                                       beta, Y, ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
void axpby_f32(int n, int ncols, float alpha, const float *X, int ldx, float beta, float *Y,
               int ldy, cudaStream_t st) {
    if (n <= 0 || ncols <= 0) return;
    k_axpby<float><<<grid_for((size_t)n * ncols, 256), 256, 0, st>>>(n, ncols, alpha, X, ldx, beta,
                                                                      Y, ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_scale_cols(int n, int m, double *__restrict__ Y, int ldy,
                             const double *__restrict__ s, int inc) {
    const size_t total = (size_t)n * m;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        const double b = s[inc == 0 ? 0 : (size_t)c * inc];
        Y[i + (size_t)c * ldy] = b == 0.0 ? 0.0 : b * Y[i + (size_t)c * ldy];
    }
}
void scale_columns_strided(int n, int m, double *Y, int ldy, const double *s, int inc,
                           cudaStream_t st) {
    if (n <= 0 || m <= 0) return;
    k_scale_cols<<<grid_for((size_t)n * m, 256), 256, 0, st>>>(n, m, Y, ldy, s, inc);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
void scale_columns(int n, int k, double *X, int ldx, const double *s, cudaStream_t st) {
    scale_columns_strided(n, k, X, ldx, s, 1, st);
}

// ---------------------------------------------------------------- X * C
// Tile TM rows x TN columns of Y per block, NT threads; thread t owns row
// t % TM and TN / (NT / TM) consecutive columns.  X and C tiles are staged
// through shared memory in chunks of TK.
template <int TM, int TN, int TK, int NT>
__global__ void __launch_bounds__(NT)
k_lincomb(int n, int k, int m, const double *__restrict__ X, int ldx, const double *__restrict__ C,
          int ldc, double *__restrict__ Y, int ldy, const double *__restrict__ beta, int incb,
          double alpha) {
    constexpr int G = NT / TM;      // column groups
    constexpr int CPT = TN / G;     // columns per thread
    __shared__ double Xs[TK][TM];
    __shared__ double Cs[TK][TN + 1];
    const int t = threadIdx.x;
    const int r = t % TM, g = t / TM;
    const int row0 = blockIdx.x * TM, col0 = blockIdx.y * TN;
    double acc[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) acc[j] = 0.0;
    for (int k0 = 0; k0 < k; k0 += TK) {
        for (int idx = t; idx < TK * TM; idx += NT) {
            const int l = idx / TM, rr = idx % TM;
            const int gr = row0 + rr, gl = k0 + l;
            Xs[l][rr] = (gr < n && gl < k) ? X[gr + (size_t)gl * ldx] : 0.0;
        }
        for (int idx = t; idx < TK * TN; idx += NT) {
            const int l = idx % TK, jj = idx / TK;
            const int gl = k0 + l, gc = col0 + jj;
            Cs[l][jj] = (gl < k && gc < m) ? C[gl + (size_t)gc * ldc] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int l = 0; l < TK; ++l) {
            const double x = Xs[l][r];
#pragma unroll
            for (int j = 0; j < CPT; ++j) acc[j] = fma(x, Cs[l][g * CPT + j], acc[j]);
        }
        __syncthreads();
    }
    const int gr = row0 + r;
    if (gr < n) {
#pragma unroll
        for (int j = 0; j < CPT; ++j) {
            const int gc = col0 + g * CPT + j;
            if (gc < m) {
                double y = alpha * acc[j];
                if (beta != nullptr) {
                    const double b = beta[incb == 0 ? 0 : (size_t)gc * incb];
                    if (b != 0.0) y = fma(b, Y[gr + (size_t)gc * ldy], y);
                }
                Y[gr + (size_t)gc * ldy] = y;
            }
        }
    }
}

// The same product for outputs too small to fill the part with 64-row tiles
// (the s x s products of the dense eigensolver, the projected-space vectors of
// ComputeP, blocks of a few thousand rows): 16 x TN tiles, one output per
// thread, the next TK columns of X and rows of C loaded into registers while
// the current ones are multiplied.  An SM issues two FP64 FMAs per clock, so
// what counts is that every SM gets the same number of outputs and that its
// warps do not wait for loads (before, 64-thread tiles with two warps per SM,
// against now: s = 180 51 -> 16.5 us, where the FP64 rate is 9.7; 200 x 160 x
// 20 43 -> 10.4; 16384 x 60 x 4 33 -> 10.4; 16384 x 180 x 20 179 -> 103).
template <int TN>
__global__ void __launch_bounds__(16 * TN)
k_lincomb_small(int n, int k, int m, const double *__restrict__ X, int ldx,
                const double *__restrict__ C, int ldc, double *__restrict__ Y, int ldy,
                const double *__restrict__ beta, int incb, double alpha) {
    constexpr int TK = 32, NT = 16 * TN;
    constexpr int NX = (16 * TK + NT - 1) / NT, NC = (TN * TK + NT - 1) / NT;
    __shared__ double Xs[TK][16];
    __shared__ double Cs[TN][TK + 1];
    const int t = threadIdx.x, r = t % 16, j = t / 16;
    const int row0 = blockIdx.x * 16, col0 = blockIdx.y * TN;
    double xq[NX], cq[NC];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < NX; ++q) {
            const int idx = t + q * NT, l = idx / 16, rr = idx % 16;
            xq[q] = (l < TK && k0 + l < k && row0 + rr < n)
                        ? __ldg(X + row0 + rr + (size_t)(k0 + l) * ldx)
                        : 0.0;
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            const int idx = t + q * NT, l = idx % TK, jj = idx / TK;
            cq[q] = (jj < TN && k0 + l < k && col0 + jj < m)
                        ? __ldg(C + k0 + l + (size_t)(col0 + jj) * ldc)
                        : 0.0;
        }
    };
    double acc = 0.0;
    fetch(0);
    for (int k0 = 0; k0 < k; k0 += TK) {
#pragma unroll
        for (int q = 0; q < NX; ++q) {
            const int idx = t + q * NT;
            if (idx < 16 * TK) Xs[idx / 16][idx % 16] = xq[q];
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            const int idx = t + q * NT;
            if (idx < TN * TK) Cs[idx / TK][idx % TK] = cq[q];
        }
        __syncthreads();
        fetch(k0 + TK);
        const int kc = min(TK, k - k0);
        if (kc == TK) {
#pragma unroll
            for (int l = 0; l < TK; ++l) acc = fma(Xs[l][r], Cs[j][l], acc);
        } else {
            for (int l = 0; l < kc; ++l) acc = fma(Xs[l][r], Cs[j][l], acc);
        }
        __syncthreads();
    }
    const int gr = row0 + r, gc = col0 + j;
    if (gr < n && gc < m) {
        double y = alpha * acc;
        if (beta != nullptr) {
            const double b = beta[incb == 0 ? 0 : (size_t)gc * incb];
            if (b != 0.0) y = fma(b, Y[gr + (size_t)gc * ldy], y);
        }
        Y[gr + (size_t)gc * ldy] = y;
    }
}

static int ceil_div(int a, int b) { return (a + b - 1) / b; }
// Column tile of at most 32 columns, a multiple of q, that splits w evenly
// (w = 40: two tiles of 20, where 32 + 8 would multiply 24 idle columns:
// 262144 x 180 x 40 5.19 -> 3.27 ms, 1.15 TFLOP/s).
static int even_tile(int w, int q) { return ceil_div(ceil_div(w, ceil_div(w, 32)), q) * q; }

void lincomb(int n, int k, int m, const double *X, int ldx, const double *C, int ldc, double *Y,
             int ldy, const double *beta_dev, int incb, cudaStream_t st, double alpha) {
    if (n <= 0 || m <= 0) return;
    if (k <= 0) {  // Y = Y diag(beta)
        if (beta_dev == nullptr) {
            for (int c = 0; c < m; ++c)
                GCGE_CUDA(cudaMemsetAsync(Y + (size_t)c * ldy, 0, sizeof(double) * n, st));
        } else {
            scale_columns_strided(n, m, Y, ldy, beta_dev, incb, st);  // incb 0 = scalar
        }
        return;
    }
    // 64-row tiles once they give every SM eight or more (an SM's share then
    // varies by an eighth at most); below that 16-row tiles, with the column
    // tile whose largest share of one SM is smallest
    const int sms = num_sms();
    const int tn = even_tile(m, 4);
    if ((long long)ceil_div(n, 64) * ceil_div(m, tn) >= 8LL * sms) {
        dim3 grid(ceil_div(n, 64), ceil_div(m, tn));
        switch (tn) {
#define GCGE_LC_CASE(W)                                                                         \
    case W:                                                                                    \
        k_lincomb<64, W, 16, 256><<<grid, 256, 0, st>>>(n, k, m, X, ldx, C, ldc, Y, ldy, beta_dev, \
                                                        incb, alpha);                          \
        break;
            GCGE_LC_CASE(4) GCGE_LC_CASE(8) GCGE_LC_CASE(12) GCGE_LC_CASE(16) GCGE_LC_CASE(20)
            GCGE_LC_CASE(24) GCGE_LC_CASE(28) GCGE_LC_CASE(32)
#undef GCGE_LC_CASE
            default: break;
        }
    } else {
        int best = 4;
        long long best_share = -1;
        for (int w = 4; w <= 32; w += 4) {
            const long long tiles = (long long)ceil_div(n, 16) * ceil_div(m, w);
            const long long share = (tiles + sms - 1) / sms * w;
            if (best_share < 0 || share <= best_share) best_share = share, best = w;
        }
        dim3 grid(ceil_div(n, 16), ceil_div(m, best));
        switch (best) {
#define GCGE_LC_CASE(W)                                                                          \
    case W:                                                                                     \
        k_lincomb_small<W><<<grid, 16 * W, 0, st>>>(n, k, m, X, ldx, C, ldc, Y, ldy, beta_dev, incb, \
                                                    alpha);                                     \
        break;
            GCGE_LC_CASE(4) GCGE_LC_CASE(8) GCGE_LC_CASE(12) GCGE_LC_CASE(16) GCGE_LC_CASE(20)
            GCGE_LC_CASE(24) GCGE_LC_CASE(28) GCGE_LC_CASE(32)
#undef GCGE_LC_CASE
            default: break;
        }
    }
    GCGE_CHECK_LAUNCH();
    count_launch();
}

// ---------------------------------------------------------------- Q^T P
// Block (chunk, mt, wt) accumulates the tile (mt, wt) of Q^T P, ta x tb
// outputs, over its row chunk.  Thread t owns row t % ta of the tile and CPT
// of its columns, ng apart (ng ta <= NT threads work).  ta and tb are not
// fixed: an FMA occupies a scheduler's FP64 unit for 64 clocks, so the tile
// that leaves the fewest lanes idle wins (fixed 32 x 24 tiles spent 48% of
// the FMAs of a 20 x 20 product on padding).  Before -> now, with n = 262144:
// 20 x 20 387 -> 226 us, 180 x 20 2.05 -> 1.79 ms, 180 x 40 5.49 -> 3.58 ms
// (1.05 TFLOP/s).
constexpr int kGT = 32;  // rows of Q and P staged at a time
template <int CPT>
__global__ void __launch_bounds__(512)
k_gram_chunk(int n, int m, int w, const double *__restrict__ Q, int ldq,
             const double *__restrict__ P, int ldp, double *__restrict__ part, int rows_per_chunk,
             int ta, int tb, int ng) {
    extern __shared__ double gsm[];
    double *Qs = gsm, *Ps = gsm + kGT * (ta + 1);
    const int t = threadIdx.x, nt = blockDim.x;
    const int a0 = blockIdx.y * ta, b0 = blockIdx.z * tb;
    const int na = min(ta, m - a0), nb = min(tb, w - b0);
    const int r_begin = blockIdx.x * rows_per_chunk;
    const int r_end = min(n, r_begin + rows_per_chunk);
    const int a = t % ta, g = t / ta;
    const bool work = g < ng;
    int pb[CPT];
    double acc[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
        pb[j] = min(g + j * ng, tb - 1);
        acc[j] = 0.0;
    }
    for (int r0 = r_begin; r0 < r_end; r0 += kGT) {
        const int i = t % kGT, gi = r0 + i;
#pragma unroll 4
        for (int cc = t / kGT; cc < ta; cc += nt / kGT)
            Qs[i * (ta + 1) + cc] = (gi < r_end && cc < na) ? Q[gi + (size_t)(a0 + cc) * ldq] : 0.0;
#pragma unroll 4
        for (int cc = t / kGT; cc < tb; cc += nt / kGT)
            Ps[i * (tb + 1) + cc] = (gi < r_end && cc < nb) ? P[gi + (size_t)(b0 + cc) * ldp] : 0.0;
        __syncthreads();
        if (work) {
            const double *q = Qs + a, *p = Ps;
#pragma unroll 8
            for (int l = 0; l < kGT; ++l, q += ta + 1, p += tb + 1) {
                const double x = *q;
#pragma unroll
                for (int j = 0; j < CPT; ++j) acc[j] = fma(x, p[pb[j]], acc[j]);
            }
        }
        __syncthreads();
    }
    const size_t base = (size_t)blockIdx.x * m * w;
#pragma unroll
    for (int j = 0; j < CPT; ++j)
        if (work && a < na && g + j * ng < nb)
            part[base + a0 + a + (size_t)(b0 + g + j * ng) * m] = acc[j];
}

// 32 x 32 tiles, a fixed launch shape with a fixed name (GCGE_GramNoAlloc):
// thread t owns row t % 32 of the tile and four columns.
__global__ void __launch_bounds__(256)
k_gram(int n, int m, int w, const double *__restrict__ Q, int ldq, const double *__restrict__ P,
       int ldp, double *__restrict__ part, int rows_per_chunk) {
    __shared__ double Qs[kGT][kGT + 1];
    __shared__ double Ps[kGT][kGT + 1];
    const int t = threadIdx.x;
    const int a = t % kGT, g = t / kGT;
    const int a0 = blockIdx.y * kGT, b0 = blockIdx.z * kGT;
    const int r_begin = blockIdx.x * rows_per_chunk;
    const int r_end = min(n, r_begin + rows_per_chunk);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int r0 = r_begin; r0 < r_end; r0 += kGT) {
        for (int idx = t; idx < kGT * kGT; idx += 256) {
            const int i = idx % kGT, cc = idx / kGT;
            const int gi = r0 + i;
            Qs[i][cc] = (gi < r_end && a0 + cc < m) ? Q[gi + (size_t)(a0 + cc) * ldq] : 0.0;
            Ps[i][cc] = (gi < r_end && b0 + cc < w) ? P[gi + (size_t)(b0 + cc) * ldp] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int i = 0; i < kGT; ++i) {
            const double q = Qs[i][a];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = fma(q, Ps[i][g * 4 + j], acc[j]);
        }
        __syncthreads();
    }
    const size_t base = (size_t)blockIdx.x * m * w;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int ga = a0 + a, gb = b0 + g * 4 + j;
        if (ga < m && gb < w) part[base + ga + (size_t)gb * m] = acc[j];
    }
}

// Split-k partial sums in a fixed order: a block sums O outputs, thread
// (o, grp) the partials grp, grp + NG, ... of output o (NG = 256 / O), then the
// groups are added in a fixed tree.  FP64 additions bound it (two per clock
// and SM), so many partials are spread over many blocks of 8 outputs; one
// thread per output walked 228 partials in 24 us.
template <int O>
__device__ __forceinline__ void reduce_chunks(const double *__restrict__ part, int chunks, int m,
                                              int w, double *__restrict__ C, int ldc) {
    constexpr int NG = 256 / O;
    __shared__ double red[8][O];
    const int total = m * w;
    const int o = threadIdx.x % O, grp = threadIdx.x / O, warp = threadIdx.x >> 5;
    for (int e0 = blockIdx.x * O; e0 < total; e0 += gridDim.x * O) {
        const int e = e0 + o;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        if (e < total) {
            int c = grp;
            for (; c + 3 * NG < chunks; c += 4 * NG) {
                s0 += part[(size_t)c * total + e];
                s1 += part[(size_t)(c + NG) * total + e];
                s2 += part[(size_t)(c + 2 * NG) * total + e];
                s3 += part[(size_t)(c + 3 * NG) * total + e];
            }
            for (; c < chunks; c += NG) s0 += part[(size_t)c * total + e];
        }
        double s = (s0 + s1) + (s2 + s3);
#pragma unroll
        for (int d = O; d < 32; d *= 2) s += __shfl_xor_sync(0xffffffffu, s, d);
        if ((threadIdx.x & 31) < O) red[warp][o] = s;
        __syncthreads();
        if (threadIdx.x < O && e < total)
            C[e % m + (size_t)(e / m) * ldc] = ((red[0][o] + red[1][o]) + (red[2][o] + red[3][o])) +
                                               ((red[4][o] + red[5][o]) + (red[6][o] + red[7][o]));
        __syncthreads();
    }
}
__global__ void __launch_bounds__(256)
k_reduce_chunks(const double *__restrict__ part, int chunks, int m, int w,
                double *__restrict__ C, int ldc) {
    if (chunks > 64) reduce_chunks<8>(part, chunks, m, w, C, ldc);
    else reduce_chunks<32>(part, chunks, m, w, C, ldc);
}
int reduce_chunks_blocks(int chunks, int outputs, int sms) {
    return std::max(1, std::min(ceil_div(outputs, chunks > 64 ? 8 : 32), 8 * sms));
}

// Short contractions (the projected space: a few hundred rows): 16 x TN tiles,
// one output per thread, the rows split over the CTAs of a cluster, whose
// partial tiles are added through distributed shared memory in rank order, so
// there are no partials in global memory and no second kernel.  As in
// k_lincomb_small the FP64 units bound it once every SM has work (200 rows,
// 140 x 20 outputs: 37 us in ten 256-thread blocks before, 6.3 us now;
// s = 180: 36 -> 16.4 us).
template <int TN>
__global__ void __launch_bounds__(16 * TN)
k_gram_small(int n, int m, int w, const double *__restrict__ Q, int ldq,
             const double *__restrict__ P, int ldp, double *__restrict__ C, int ldc) {
    constexpr int NT = 16 * TN;
    constexpr int NQ = (16 * kGT + NT - 1) / NT, NP = (TN * kGT + NT - 1) / NT;
    __shared__ double Qs[16][kGT + 1];
    __shared__ double Ps[TN][kGT + 1];
    __shared__ double tile[NT];
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int cs = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int t = threadIdx.x, a = t % 16, b = t / 16;
    const int a0 = blockIdx.y * 16, b0 = blockIdx.z * TN;
    const int rpc = (n + cs - 1) / cs;
    const int r_begin = min(n, rank * rpc), r_end = min(n, r_begin + rpc);
    double qq[NQ], pq[NP];
    auto fetch = [&](int r0) {
#pragma unroll
        for (int u = 0; u < NQ; ++u) {
            const int idx = t + u * NT, i = r0 + idx % kGT, cc = idx / kGT;
            qq[u] = (cc < 16 && i < r_end && a0 + cc < m) ? __ldg(Q + i + (size_t)(a0 + cc) * ldq)
                                                         : 0.0;
        }
#pragma unroll
        for (int u = 0; u < NP; ++u) {
            const int idx = t + u * NT, i = r0 + idx % kGT, cc = idx / kGT;
            pq[u] = (cc < TN && i < r_end && b0 + cc < w) ? __ldg(P + i + (size_t)(b0 + cc) * ldp)
                                                         : 0.0;
        }
    };
    double acc = 0.0;
    fetch(r_begin);
    for (int r0 = r_begin; r0 < r_end; r0 += kGT) {
#pragma unroll
        for (int u = 0; u < NQ; ++u) {
            const int idx = t + u * NT;
            if (idx < 16 * kGT) Qs[idx / kGT][idx % kGT] = qq[u];
        }
#pragma unroll
        for (int u = 0; u < NP; ++u) {
            const int idx = t + u * NT;
            if (idx < TN * kGT) Ps[idx / kGT][idx % kGT] = pq[u];
        }
        __syncthreads();
        fetch(r0 + kGT);
        const int rc = min(kGT, r_end - r0);
        if (rc == kGT) {
#pragma unroll
            for (int i = 0; i < kGT; ++i) acc = fma(Qs[a][i], Ps[b][i], acc);
        } else {
            for (int i = 0; i < rc; ++i) acc = fma(Qs[a][i], Ps[b][i], acc);
        }
        __syncthreads();
    }
    if (cs > 1) {
        tile[t] = acc;
        cl.sync();
        // CTA `rank` adds the outputs [rank NT / cs, (rank + 1) NT / cs) (NT is a
        // multiple of 64, cs 1, 2, 4 or 8)
        const int per = NT / cs, o = rank * per + t;
        if (t < per) {
            double s = 0.0;
            for (int c = 0; c < cs; ++c) s += *cl.map_shared_rank(tile + o, c);
            const int ga = a0 + o % 16, gb = b0 + o / 16;
            if (ga < m && gb < w) C[ga + (size_t)gb * ldc] = s;
        }
        cl.sync();  // no CTA leaves while another reads its tile
    } else if (a0 + a < m && b0 + b < w) {
        C[a0 + a + (size_t)(b0 + b) * ldc] = acc;
    }
}

// The shape of a Gram product: `small` the cluster kernel with tiles 16 x tb
// over clusters of cs CTAs, else tiles ta x tb of nt threads with cpt outputs
// each over row chunks.
struct GramPlan {
    bool small;
    int ta, tb, nt, ng, cpt, cs, chunks;
};
static GramPlan gram_plan(int n, int m, int w) {
    const int sms = num_sms();
    GramPlan g{false, 1, 1, 128, 1, 1, 1, 1};
    // chunked form: even tiles of at most 64 x 32, and the threads and outputs
    // per thread that leave the fewest idle lanes on the four schedulers
    g.ta = ceil_div(m, ceil_div(m, 64));
    g.tb = ceil_div(w, ceil_div(w, 32));
    int lanes = 0;
    for (int cpt = 1; cpt <= 8; ++cpt) {
        const int ng = ceil_div(g.tb, cpt), nt = ceil_div(g.ta * ng, 128) * 128;
        if (nt > 512) continue;
        if (lanes == 0 || nt * cpt < lanes || (nt * cpt == lanes && nt >= 256)) {
            lanes = nt * cpt;
            g.nt = nt;
            g.ng = ng;
            g.cpt = cpt;
        }
    }
    // about four blocks of 256 threads per SM, each SM the same number of them
    const int tiles = ceil_div(m, g.ta) * ceil_div(w, g.tb);
    g.chunks = std::min(std::max(1, sms * (1024 / g.nt) / tiles), ceil_div(n, kGT));
    // FP64 clocks of the busiest SM (two FMAs per clock); a chunked product
    // pays for a second launch, the cluster form for two cluster barriers.
    // The cluster form is for short contractions: its tiles read Q and P from
    // L2 again for every 16 columns, with few warps to hide it.
    const long long rows = (long long)ceil_div(ceil_div(n, g.chunks), kGT) * kGT;
    const long long blocks = (long long)tiles * ceil_div(n, (int)rows);
    long long best = (blocks + sms - 1) / sms * lanes * rows / 2 + 8000;
    if (n > 1024) return g;
    for (int tb = 4; tb <= 32; tb += 4)
        for (int cs = 1; cs <= 8; cs *= 2) {
            // a CTA's chain of FMAs takes 90 clocks a row (measured), unless the
            // SM's share of CTAs keeps its FP64 units busier than that
            const int ctas = ceil_div(m, 16) * ceil_div(w, tb) * cs;
            const long long lanes_sm = (long long)ceil_div(ctas, sms) * ceil_div(16 * tb, 128) * 64;
            const long long cost =
                ceil_div(n, cs) * std::max(90LL, lanes_sm) + 600 + (cs > 1 ? 1000 : 0);
            if (cost < best) {
                best = cost;
                g.small = true;
                g.cs = cs;
                g.tb = tb;
            }
        }
    return g;
}
size_t gram_scratch_elems(int n, int m, int w) {
    if (m <= 0 || w <= 0) return 0;
    return (size_t)gram_plan(std::max(n, 1), m, w).chunks * m * w;
}

template <int TN>
static void launch_gram_small(int cs, int n, int m, int w, const double *Q, int ldq,
                              const double *P, int ldp, double *C, int ldc, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs, ceil_div(m, 16), ceil_div(w, TN));
    cfg.blockDim = dim3(16 * TN);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    GCGE_CUDA(cudaLaunchKernelEx(&cfg, k_gram_small<TN>, n, m, w, Q, ldq, P, ldp, C, ldc));
}

void gram(int n, int m, int w, const double *Q, int ldq, const double *P, int ldp, double *C,
          int ldc, double *scratch, size_t scratch_elems, cudaStream_t st) {
    if (m <= 0 || w <= 0) return;
    if (n <= 0) {
        for (int b = 0; b < w; ++b)
            GCGE_CUDA(cudaMemsetAsync(C + (size_t)b * ldc, 0, sizeof(double) * m, st));
        return;
    }
    const GramPlan g = gram_plan(n, m, w);
    if (g.small) {
        switch (g.tb) {
#define GCGE_GR_CASE(W)                                                              \
    case W:                                                                         \
        launch_gram_small<W>(g.cs, n, m, w, Q, ldq, P, ldp, C, ldc, st);             \
        break;
            GCGE_GR_CASE(4) GCGE_GR_CASE(8) GCGE_GR_CASE(12) GCGE_GR_CASE(16) GCGE_GR_CASE(20)
            GCGE_GR_CASE(24) GCGE_GR_CASE(28) GCGE_GR_CASE(32)
#undef GCGE_GR_CASE
            default: break;
        }
        count_launch();
        return;
    }
    // the scratch may have been sized for another shape: fewer, longer chunks
    GCGE_REQUIRE((size_t)m * w <= scratch_elems, GCGE_ERR_ARG, "gram: scratch too small");
    const int chunks = (int)std::min<size_t>(g.chunks, scratch_elems / ((size_t)m * w));
    const int rpc = ceil_div(ceil_div(n, chunks), kGT) * kGT;
    const int nchunks = ceil_div(n, rpc);
    const dim3 grid(nchunks, ceil_div(m, g.ta), ceil_div(w, g.tb));
    const size_t smem = sizeof(double) * kGT * (g.ta + g.tb + 2);  // at most 25 KB
    switch (g.cpt) {
#define GCGE_GR_CASE(W)                                                                      \
    case W:                                                                                 \
        k_gram_chunk<W><<<grid, g.nt, smem, st>>>(n, m, w, Q, ldq, P, ldp, scratch, rpc, g.ta, \
                                                  g.tb, g.ng);                              \
        break;
        GCGE_GR_CASE(1) GCGE_GR_CASE(2) GCGE_GR_CASE(3) GCGE_GR_CASE(4) GCGE_GR_CASE(5)
        GCGE_GR_CASE(6) GCGE_GR_CASE(7) GCGE_GR_CASE(8)
#undef GCGE_GR_CASE
        default: break;
    }
    GCGE_CHECK_LAUNCH();
    k_reduce_chunks<<<reduce_chunks_blocks(nchunks, m * w, num_sms()), 256, 0, st>>>(
        scratch, nchunks, m, w, C, ldc);
    GCGE_CHECK_LAUNCH();
    count_launch(2);
}

// ---------------------------------------------------------------- column dots
__global__ void __launch_bounds__(256)
k_coldot(int n, int k, const double *__restrict__ X, int ldx, const double *__restrict__ Y, int ldy,
         double *__restrict__ part, int rows_per_chunk) {
    __shared__ double red[8];
    const int c = blockIdx.y;
    const int r_begin = blockIdx.x * rows_per_chunk;
    const int r_end = min(n, r_begin + rows_per_chunk);
    double s = 0.0;
    for (int i = r_begin + threadIdx.x; i < r_end; i += 256)
        s = fma(X[i + (size_t)c * ldx], Y[i + (size_t)c * ldy], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tsum = 0.0;
        for (int i = 0; i < 8; ++i) tsum += red[i];
        part[(size_t)blockIdx.x * k + c] = tsum;
    }
}

void coldot(int n, int k, const double *X, int ldx, const double *Y, int ldy, double *out,
            double *scratch, size_t scratch_elems, cudaStream_t st) {
    if (k <= 0) return;
    int chunks = std::max(1, std::min((n + 2047) / 2048, (2 * num_sms() + k - 1) / k));
    while ((size_t)chunks * k > scratch_elems && chunks > 1) chunks /= 2;
    GCGE_REQUIRE((size_t)chunks * k <= scratch_elems, GCGE_ERR_ARG, "coldot: scratch too small");
    const int rpc = (n + chunks - 1) / chunks;
    dim3 grid(chunks, k);
    k_coldot<<<grid, 256, 0, st>>>(n, k, X, ldx, Y, ldy, scratch, rpc);
    GCGE_CHECK_LAUNCH();
    count_launch();
    reduce_partials(scratch, chunks, k, k, out, st);
}

__global__ void k_reduce_partials(const double *__restrict__ part, int nblocks, int kmax,
                                  double *__restrict__ out) {
    __shared__ double red[256];
    const int c = blockIdx.x;
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 256) s += part[(size_t)b * kmax + c];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = red[0];
}

void reduce_partials(const double *partial, int nblocks, int kmax, int k, double *out,
                     cudaStream_t st) {
    if (k <= 0) return;
    k_reduce_partials<<<k, 256, 0, st>>>(partial, nblocks, kmax, out);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

// ---------------------------------------------------------------- helpers
template <typename S, typename D>
__global__ void k_convert(int n, int k, const S *__restrict__ X, int ldx, D *__restrict__ Y,
                          int ldy) {
    const size_t total = (size_t)n * k;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        Y[i + (size_t)c * ldy] = (D)X[i + (size_t)c * ldx];
    }
}
void copy_f64_to_f32(int n, int k, const double *X, int ldx, float *Y, int ldy, cudaStream_t st) {
    if (n <= 0 || k <= 0) return;
    k_convert<double, float><<<grid_for((size_t)n * k, 256), 256, 0, st>>>(n, k, X, ldx, Y, ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
__global__ void k_add_f32(int n, int k, const float *__restrict__ X, int ldx, double *__restrict__ Y,
                          int ldy) {
    const size_t total = (size_t)n * k;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        Y[i + (size_t)c * ldy] += (double)X[i + (size_t)c * ldx];
    }
}
void add_f32_to_f64(int n, int k, const float *X, int ldx, double *Y, int ldy, cudaStream_t st) {
    if (n <= 0 || k <= 0) return;
    k_add_f32<<<grid_for((size_t)n * k, 256), 256, 0, st>>>(n, k, X, ldx, Y, ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
void copy_f32_to_f64(int n, int k, const float *X, int ldx, double *Y, int ldy, cudaStream_t st) {
    if (n <= 0 || k <= 0) return;
    k_convert<float, double><<<grid_for((size_t)n * k, 256), 256, 0, st>>>(n, k, X, ldx, Y, ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__global__ void k_fill_uniform(int n, int k, double *__restrict__ X, int ldx,
                               unsigned long long seed) {
    const size_t total = (size_t)n * k;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        const unsigned long long z = mix64(seed * 0x9E3779B97F4A7C15ULL + t + 1);
        X[i + (size_t)c * ldx] = (double)(z >> 11) * (1.0 / 9007199254740992.0);
    }
}
void fill_uniform(int n, int k, double *X, int ldx, unsigned long long seed, cudaStream_t st) {
    if (n <= 0 || k <= 0) return;
    k_fill_uniform<<<grid_for((size_t)n * k, 256), 256, 0, st>>>(n, k, X, ldx, seed);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_gather_cols(int n, int k, const double *__restrict__ X, int ldx,
                              const int *__restrict__ idx, double *__restrict__ Y, int ldy) {
    const size_t total = (size_t)n * k;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        Y[i + (size_t)c * ldy] = X[i + (size_t)idx[c] * ldx];
    }
}
void gather_columns(int n, int k, const double *X, int ldx, const int *idx, double *Y, int ldy,
                    cudaStream_t st) {
    if (n <= 0 || k <= 0) return;
    k_gather_cols<<<grid_for((size_t)n * k, 256), 256, 0, st>>>(n, k, X, ldx, idx, Y, ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_identity(int n, double *__restrict__ X, int ldx) {
    const size_t total = (size_t)n * n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        X[i + (size_t)c * ldx] = i == c ? 1.0 : 0.0;
    }
}
void set_identity(int n, double *X, int ldx, cudaStream_t st) {
    if (n <= 0) return;
    k_identity<<<grid_for((size_t)n * n, 256), 256, 0, st>>>(n, X, ldx);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_fill(size_t count, double *__restrict__ X, double v) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < count;
         t += (size_t)gridDim.x * blockDim.x)
        X[t] = v;
}
void fill_value(size_t count, double *X, double v, cudaStream_t st) {
    if (count == 0) return;
    k_fill<<<grid_for(count, 256), 256, 0, st>>>(count, X, v);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

}  // namespace gcge

namespace gcge {

// max |C_ij| into *out, which may be page-locked host memory (the callers wait
// for the stream before they read it: no copy of its own).  On the bits, which
// order as the magnitudes do, a NaN above all: an FP64 comparison occupies a
// scheduler for 64 clocks, and a block of them made this 9 us for 240 entries.
__global__ void k_absmax(int m, int w, const double *__restrict__ C, int ldc, double *out) {
    __shared__ unsigned long long red[32];
    unsigned long long v = 0;
    for (int e = threadIdx.x; e < m * w; e += blockDim.x) {
        const unsigned long long a =
            (unsigned long long)__double_as_longlong(C[(e % m) + (size_t)(e / m) * ldc]) << 1;
        v = a > v ? a : v;
    }
    auto warp_max = [](unsigned long long x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long u = __shfl_xor_sync(0xffffffffu, x, o);
            x = u > x ? u : x;
        }
        return x;
    };
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = warp_max(threadIdx.x < (blockDim.x + 31) / 32 ? red[threadIdx.x] : 0ull);
        if (threadIdx.x == 0) *out = __longlong_as_double((long long)(v >> 1));
    }
}
void absmax(int m, int w, const double *C, int ldc, double *out, cudaStream_t st) {
    const int threads = (int)std::min<long long>(1024, ((long long)m * w + 31) / 32 * 32);
    k_absmax<<<1, std::max(threads, 32), 0, st>>>(m, w, C, ldc, out);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_zero_rows(int m, int k, double *__restrict__ X, int ldx,
                            const int *__restrict__ mask) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m * k; e += gridDim.x * blockDim.x) {
        const int i = e % m, j = e / m;
        if (mask[i]) X[i + (size_t)j * ldx] = 0.0;
    }
}
void zero_rows(int m, int k, double *X, int ldx, const int *mask, cudaStream_t st) {
    if (m <= 0 || k <= 0) return;
    k_zero_rows<<<std::max(1, std::min(1024, (m * k + 255) / 256)), 256, 0, st>>>(m, k, X, ldx,
                                                                                  mask);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_transpose(int m, int k, const double *__restrict__ X, int ldx,
                            double *__restrict__ Y, int ldy) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m * k; e += gridDim.x * blockDim.x) {
        const int i = e % m, j = e / m;
        Y[j + (size_t)i * ldy] = X[i + (size_t)j * ldx];
    }
}
void transpose_copy(int m, int k, const double *X, int ldx, double *Y, int ldy, cudaStream_t st) {
    if (m <= 0 || k <= 0) return;
    k_transpose<<<std::max(1, std::min(1024, (m * k + 255) / 256)), 256, 0, st>>>(m, k, X, ldx, Y,
                                                                                  ldy);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

__global__ void k_shift(size_t count, const double *__restrict__ a, const double *__restrict__ b,
                        double sigma, double *__restrict__ y64, float *__restrict__ y32) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < count;
         t += (size_t)gridDim.x * blockDim.x) {
        const double v = fma(sigma, b[t], a[t]);
        if (y64) y64[t] = v;
        if (y32) y32[t] = (float)v;
    }
}
void shift_values(size_t count, const double *a, const double *b, double sigma, double *y64,
                  float *y32, cudaStream_t st) {
    if (count == 0) return;
    k_shift<<<grid_for(count, 256), 256, 0, st>>>(count, a, b, sigma, y64, y32);
    GCGE_CHECK_LAUNCH();
    count_launch();
}

void copy_cols(int n, int k, const double *X, int ldx, double *Y, int ldy, cudaStream_t st) {
    if (n <= 0 || k <= 0 || X == Y) return;
    GCGE_CUDA(cudaMemcpy2DAsync(Y, sizeof(double) * ldy, X, sizeof(double) * ldx,
                                sizeof(double) * n, k, cudaMemcpyDeviceToDevice, st));
}

}  // namespace gcge
