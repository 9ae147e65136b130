// Block PCG (pcg_kernel.cuh): the block conversions, the work area of a solve
// and the FP32 instantiations.
#include <algorithm>

#include "pcg_kernel.cuh"

namespace gcge {

// column-major (S, ld) <-> slice-blocked (T, kp): element (i, c) of the
// blocked block sits at ((i / 32) G + c / L) 32 L + (i % 32) L + c % L with
// L = 16 / sizeof(T), G = kp / L; rows up to the next multiple of 32 and
// columns k..kp-1 are zero.
//
// A warp converts one 16-byte column group of one slice, a row per lane: whole
// 256-byte runs of every column on one side, one 512-byte run on the other, and
// one division per 32 rows instead of two or three 64-bit ones per element
// (128^3 rows x 40 columns, FP64 to FP32 and back, 1.0 GB each: 252 and 259 us with
// those, 156 and 159 now).
template <typename S, typename T>
__global__ void __launch_bounds__(256)
k_col_to_rows(int n, int k, int kp, const S *__restrict__ X, int ldx, T *__restrict__ Y) {
    constexpr int L = 16 / (int)sizeof(T);
    const int G = kp / L, lane = threadIdx.x & 31;
    const long long units = (long long)((n + 31) / 32) * G;
    for (long long w = blockIdx.x * 8ll + (threadIdx.x >> 5); w < units; w += gridDim.x * 8ll) {
        const int s = (int)(w / G), u = (int)(w - (long long)s * G), i = s * 32 + lane;
        struct alignas(16) {
            T v[L];
        } o;
#pragma unroll
        for (int e = 0; e < L; ++e) {
            const int c = u * L + e;
            o.v[e] = (i < n && c < k) ? (T)X[i + (size_t)c * ldx] : T(0);
        }
        *reinterpret_cast<decltype(o) *>(Y + (size_t)w * 32 * L + lane * L) = o;
    }
}
// *out |= a bit for each column of X (slice-blocked, FP32) with an entry that is
// not finite.  X once at HBM speed (55 us of a 25 ms solve at 128^3 x 40); a
// kernel of its own, as the three-phase kernel has no register left for it
// (k_block_pcg<float, 20> spilled 36 bytes instead of 20).
__global__ void __launch_bounds__(256)
k_out_of_range(int n, int kp, const float *__restrict__ X, unsigned long long *out) {
    const int G = kp / 4, lane = threadIdx.x & 31;
    const long long units = (long long)((n + 31) / 32) * G;
    unsigned long long bits = 0;
    for (long long w = blockIdx.x * 8ll + (threadIdx.x >> 5); w < units; w += gridDim.x * 8ll) {
        const int s = (int)(w / G), u = (int)(w - (long long)s * G);
        const float4 v = *reinterpret_cast<const float4 *>(X + (size_t)w * 128 + lane * 4);
        if (s * 32 + lane >= n) continue;
        const unsigned bad = (isfinite(v.x) ? 0u : 1u) | (isfinite(v.y) ? 0u : 2u) |
                             (isfinite(v.z) ? 0u : 4u) | (isfinite(v.w) ? 0u : 8u);
        bits |= (unsigned long long)bad << (4 * u);
    }
    if (bits) atomicOr(out, bits);
}
// add: Y += X.  On an indefinite operator a column of the FP32 correction can
// leave the range of its type (a nearly vanishing p^T S p); such a column of Y
// (its bit in *skip) stays as it was, whole, instead of spoiling the block it
// belongs to, and *report tells the host.
template <typename T, typename D>
__global__ void __launch_bounds__(256)
k_rows_to_col(int n, int k, int kp, const T *__restrict__ X, D *__restrict__ Y, int ldy, int add,
              const unsigned long long *skip, unsigned long long *report) {
    constexpr int L = 16 / (int)sizeof(T);
    const unsigned long long out = skip ? *skip : 0ull;
    if (report && out && blockIdx.x == 0 && threadIdx.x == 0) *report = out;
    const int G = kp / L, used = (k + L - 1) / L, lane = threadIdx.x & 31;
    const long long units = (long long)((n + 31) / 32) * used;
    for (long long w = blockIdx.x * 8ll + (threadIdx.x >> 5); w < units; w += gridDim.x * 8ll) {
        const int s = (int)(w / used), u = (int)(w - (long long)s * used), i = s * 32 + lane;
        struct alignas(16) Pack {
            T v[L];
        };
        const Pack q = *reinterpret_cast<const Pack *>(X + ((size_t)s * G + u) * 32 * L + lane * L);
        if (i >= n) continue;
#pragma unroll
        for (int e = 0; e < L; ++e) {
            const int c = u * L + e;
            if (c >= k || ((out >> c) & 1ull)) continue;
            const D v = (D)q.v[e];
            D &y = Y[i + (size_t)c * ldy];
            y = add ? y + v : v;
        }
    }
}

void mark_out_of_range(int n, int kp, const float *X, unsigned long long *out, cudaStream_t st) {
    const long long units = (long long)((n + 31) / 32) * (kp / 4);
    const int g = (int)std::max(1ll, std::min((units + 7) / 8, 16ll * device_sms()));
    k_out_of_range<<<g, 256, 0, st>>>(n, kp, X, out);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
template <typename S, typename T>
void col_to_rows(int n, int k, int kp, const S *X, int ldx, T *Y, cudaStream_t st) {
    const long long units = (long long)((n + 31) / 32) * (kp / (16 / (int)sizeof(T)));
    const int g = (int)std::max(1ll, std::min((units + 7) / 8, 16ll * device_sms()));
    k_col_to_rows<S, T><<<g, 256, 0, st>>>(n, k, kp, X, ldx, Y);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
template <typename T, typename D>
void rows_to_col(int n, int k, int kp, const T *X, D *Y, int ldy, bool add, cudaStream_t st,
                 const unsigned long long *out, unsigned long long *report) {
    constexpr int L = 16 / (int)sizeof(T);
    const long long units = (long long)((n + 31) / 32) * ((k + L - 1) / L);
    const int g = (int)std::max(1ll, std::min((units + 7) / 8, 16ll * device_sms()));
    k_rows_to_col<T, D><<<g, 256, 0, st>>>(n, k, kp, X, Y, ldy, add ? 1 : 0, out, report);
    GCGE_CHECK_LAUNCH();
    count_launch();
}
template void col_to_rows<double, double>(int, int, int, const double *, int, double *, cudaStream_t);
template void col_to_rows<double, float>(int, int, int, const double *, int, float *, cudaStream_t);
template void rows_to_col<double, double>(int, int, int, const double *, double *, int, bool,
                                          cudaStream_t, const unsigned long long *, unsigned long long *);
template void rows_to_col<float, double>(int, int, int, const float *, double *, int, bool,
                                         cudaStream_t, const unsigned long long *, unsigned long long *);

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
        h_out.alloc(1);
        *h_out.p = 0;
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
thread_local PcgForm t_pcg_form = kPcgNone;

template void block_pcg_rows<float>(PcgWork &, const SellPattern &, const float *, const float *,
                                    float *, float *, float *, float *, int, int, int, double,
                                    double, bool, bool, cudaStream_t);

}  // namespace gcge
