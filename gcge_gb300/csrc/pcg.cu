// Block PCG (pcg_kernel.cuh): the block conversions, the work area of a solve
// and the FP32 instantiations.
#include <algorithm>

#include "pcg_kernel.cuh"

namespace gcge {

// column-major (S, ld) <-> slice-blocked (T, kp): element (i, c) of the
// blocked block sits at ((i / 32) G + c / L) 32 L + (i % 32) L + c % L with
// L = 16 / sizeof(T), G = kp / L; rows up to the next multiple of 32 and
// columns k..kp-1 are zero.
template <typename T>
__host__ __device__ __forceinline__ size_t blk_index(int i, int c, int kp) {
    constexpr int L = 16 / (int)sizeof(T);
    const int G = kp / L;
    return ((size_t)(i >> 5) * G + c / L) * (32 * L) + (size_t)(i & 31) * L + c % L;
}
template <typename S, typename T>
__global__ void k_col_to_rows(int n, int k, int kp, const S *__restrict__ X, int ldx,
                              T *__restrict__ Y) {
    constexpr int L = 16 / (int)sizeof(T);
    const int G = kp / L;
    const size_t total = (size_t)((n + 31) / 32) * 32 * kp;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        // t = ((s G + u) 32 + l) L + e
        const int e = (int)(t % L);
        const size_t q = t / L;
        const int l = (int)(q % 32);
        const size_t su = q / 32;
        const int u = (int)(su % G);
        const int i = (int)(su / G) * 32 + l, c = u * L + e;
        Y[t] = (i < n && c < k) ? (T)X[i + (size_t)c * ldx] : T(0);
    }
}
// add: Y += X where X is finite.  On an indefinite operator a column of the FP32
// correction can leave the range of its type (a nearly vanishing p^T S p); such
// a column of Y stays as it was instead of spoiling the block it belongs to.
template <typename T, typename D>
__global__ void k_rows_to_col(int n, int k, int kp, const T *__restrict__ X, D *__restrict__ Y,
                              int ldy, int add) {
    const size_t total = (size_t)n * k;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), i = (int)(t % n);
        const D v = (D)X[blk_index<T>(i, c, kp)];
        D &y = Y[i + (size_t)c * ldy];
        y = add ? (isfinite(v) ? y + v : y) : v;
    }
}

template <typename S, typename T>
void col_to_rows(int n, int k, int kp, const S *X, int ldx, T *Y, cudaStream_t st) {
    const size_t total = (size_t)((n + 31) / 32) * 32 * kp;
    const int g = (int)std::max<size_t>(1, std::min<size_t>((total + 255) / 256, 16 * device_sms()));
    k_col_to_rows<S, T><<<g, 256, 0, st>>>(n, k, kp, X, ldx, Y);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
template <typename T, typename D>
void rows_to_col(int n, int k, int kp, const T *X, D *Y, int ldy, bool add, cudaStream_t st) {
    const size_t total = (size_t)n * k;
    const int g = (int)std::max<size_t>(1, std::min<size_t>((total + 255) / 256, 16 * device_sms()));
    k_rows_to_col<T, D><<<g, 256, 0, st>>>(n, k, kp, X, Y, ldy, add ? 1 : 0);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
template void col_to_rows<double, double>(int, int, int, const double *, int, double *, cudaStream_t);
template void col_to_rows<double, float>(int, int, int, const double *, int, float *, cudaStream_t);
template void rows_to_col<double, double>(int, int, int, const double *, double *, int, bool,
                                          cudaStream_t);
template void rows_to_col<float, double>(int, int, int, const float *, double *, int, bool,
                                         cudaStream_t);

void PcgWork::timing_reset(cudaStream_t st) {
    ev_used = 0;
    launches = 0;
    kernel_ms = spmm_ms = kernel_bytes = spmm_bytes = 0.0;
    total_iters = 0;
    GCGE_CUDA(cudaMemsetAsync(stats.p, 0, sizeof(PcgStats), st));
}
void PcgWork::collect(cudaStream_t st) {
    GCGE_CUDA(cudaMemcpyAsync(h_stats.p, stats.p, sizeof(PcgStats), cudaMemcpyDeviceToHost, st));
    GCGE_CUDA(cudaStreamSynchronize(st));
    double ms = 0.0;
    for (size_t i = 0; i + 1 < ev_used; i += 2) {
        float t = 0.f;
        if (cudaEventElapsedTime(&t, ev[i], ev[i + 1]) == cudaSuccess) ms += t;
    }
    kernel_ms = ms;
    spmm_ms = (double)h_stats.p->spmm_ns * 1e-6;
    kernel_bytes = h_stats.p->kernel_bytes;
    spmm_bytes = h_stats.p->spmm_bytes;
    total_iters = (long long)h_stats.p->iters;
    if (h_stats.p->error != 0) {
        // the launch that timed out has ended; clear the flag so the next
        // solve on this work area starts clean, then report
        GCGE_CUDA(cudaMemsetAsync(&stats.p->error, 0, sizeof(int), st));
        GCGE_CUDA(cudaStreamSynchronize(st));
        throw CudaError{GCGE_ERR_CUDA, "block PCG: a grid barrier wait timed out"};
    }
}
PcgWork::~PcgWork() {
    for (auto e : ev) cudaEventDestroy(e);
}

void PcgWork::reserve(int n, int kmax_) {
    (void)n;
    kmax = std::max(kmax_, 40);
    part.alloc((size_t)4 * device_sms() * kPcgMaxCols);
    if (!sc.p) {
        sc.alloc(1);
        sync.alloc(1);
        stats.alloc(1);
        h_sc.alloc(1);
        h_stats.alloc(1);
        GCGE_CUDA(cudaMemsetAsync(stats.p, 0, sizeof(PcgStats), lib_stream()));
    }
}

int pcg_last_iters(PcgWork &wk, cudaStream_t st) {
    GCGE_CUDA(cudaMemcpyAsync(wk.h_sc.p, wk.sc.p, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
    GCGE_CUDA(cudaMemcpyAsync(wk.h_stats.p, wk.stats.p, sizeof(PcgStats), cudaMemcpyDeviceToHost,
                              st));
    GCGE_CUDA(cudaStreamSynchronize(st));
    if (wk.h_stats.p->error != 0) {
        GCGE_CUDA(cudaMemsetAsync(&wk.stats.p->error, 0, sizeof(int), st));
        GCGE_CUDA(cudaStreamSynchronize(st));
        throw CudaError{GCGE_ERR_CUDA, "block PCG: a grid barrier wait timed out"};
    }
    return wk.h_sc.p->niter;
}

thread_local PcgBarrierTest t_pcg_barrier_test;

template void block_pcg_rows<float>(PcgWork &, const SellPattern &, const float *, const float *,
                                    float *, float *, float *, float *, int, int, int, double,
                                    double, bool, bool, cudaStream_t);

}  // namespace gcge
