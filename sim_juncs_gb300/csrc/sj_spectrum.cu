// The spectrum save_field_times writes for each monitor series
// (src/disp.cpp:804, with the fft of src/data_utils.cpp:413-427): of N
// samples it takes the first N' = 2^floor(log2 N) and evaluates
//   F_k = sum_{m < N'} x_m e^{-i 2 pi m k / N},  k = -N'/2 .. N'/2 - 1,
// stored at index k mod N' (the phase step is 2 pi / N, not 2 pi / N').
// The reference does this O(N'^2) on the host per monitor.  Here a thread sums
// one bin k >= 0 of several monitors, FP64; F_{-k} is its conjugate, the
// samples being real.  The phase m k modulo N advances by an addition and
// indexes a table of e^{-i 2 pi r / N}, so a term is two FP64 operations per
// monitor, which bound the kernel (1024 monitors, 1000 samples: 0.66 ms, of
// which the FP64 pipe's 19 cycles per warp operation make 0.5; 22 ms with a
// sincospi and a 64-bit remainder per term).
#include "sj_internal.h"

namespace sj {

namespace {

constexpr int SPEC_THREADS = 64;

__global__ void k_spectrum_table(long long n, double2* __restrict__ tab) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double s, c;
    sincospi(-2.0 * (double)r / (double)n, &s, &c);
    tab[r] = make_double2(c, s);
}

// bins 0 .. np/2 of monitors R blockIdx.y .. + R - 1
template <int R>
__global__ void __launch_bounds__(SPEC_THREADS)
k_spectrum(const double* __restrict__ mon, int n_mon, unsigned n, long long np, const double2* __restrict__ tab,
           double* __restrict__ out) {
    const int ms = blockIdx.y * R;
    const long long k = (long long)blockIdx.x * SPEC_THREADS + threadIdx.x;
    if (k > np / 2) return;
    double re[R], im[R];
#pragma unroll
    for (int q = 0; q < R; ++q) re[q] = im[q] = 0.0;
    if (np > 1) {
        const unsigned step = (unsigned)k;
        unsigned r = 0;
        for (long long m = 0; m < np; ++m) {
            const double2 e = __ldg(tab + r);
            const double* x = mon + m * n_mon + ms;
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const double v = R == 1 || ms + q < n_mon ? __ldg(x + q) : 0.0;
                re[q] += v * e.x;
                im[q] += v * e.y;
            }
            r += step;
            if (r >= n) r -= n;
        }
    }
    double2* o = reinterpret_cast<double2*>(out);
#pragma unroll
    for (int q = 0; q < R; ++q) {
        if (ms + q >= n_mon) continue;
        double2* row = o + (long long)(ms + q) * np;
        if (k < np / 2 || np == 1) row[k] = make_double2(re[q], im[q]);
        if (k > 0) row[np - k] = make_double2(re[q], -im[q]);
    }
}

}  // namespace

cudaError_t launch_spectrum(const double* d_mon, int n_mon, long long n, long long np, double2* d_table, double* d_out,
                            cudaStream_t s) {
    if (n_mon < 1 || np < 1) return cudaSuccess;
    k_spectrum_table<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, d_table);
    const unsigned bins = (unsigned)((np / 2 + SPEC_THREADS) / SPEC_THREADS);
    // monitors per thread: eight share a term's table entry and index where
    // that leaves enough threads, one on a few monitors
    const auto groups = [&](int r) { return (unsigned)((n_mon + r - 1) / r); };
    if ((long long)bins * groups(8) >= 304)
        k_spectrum<8><<<dim3(bins, groups(8)), SPEC_THREADS, 0, s>>>(d_mon, n_mon, (unsigned)n, np, d_table, d_out);
    else if ((long long)bins * groups(2) >= 304)
        k_spectrum<2><<<dim3(bins, groups(2)), SPEC_THREADS, 0, s>>>(d_mon, n_mon, (unsigned)n, np, d_table, d_out);
    else
        k_spectrum<1><<<dim3(bins, groups(1)), SPEC_THREADS, 0, s>>>(d_mon, n_mon, (unsigned)n, np, d_table, d_out);
    return cudaGetLastError();
}

}  // namespace sj
