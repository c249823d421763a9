// CEP and envelope extraction from monitor series, one CUDA block per series.
//
// Restates the reference's analysis class `signal` (scripts/phases.py:94-450)
// on its default path, as the sweeps call it (signal(t, v, lowpass_inc),
// get_envelope(), get_skewness()):
//   1. t0 guess: the |v|-weighted mean index of the local maxima of v^2
//      (_guess_t0_ind, :95-105; scipy.signal.find_peaks' plateau rule);
//   2. V = 2 rfft(v rolled by -t0); repeat: f0_ind = argmax |V|, f0 = the
//      trapezoid mean frequency of |V| below 2 f0_ind (_est_f0 'avg',
//      :225-228); a sinc low-pass of growing strength when f0 is above half
//      the band or |V| has a prominent peak above 3 f0 (is_noisy, :264-276),
//      at most MAX_LOWPASS_EVALS times (:313-341);
//   3. the band where |V| exceeds CUT_ALPHA of its value at f0 (_get_freq_fwhm,
//      :107-122), the unwrapped phase there (fix_angle_seq, :63-74) and its
//      linear regression: t0_corr = -slope / 2 pi, phi = intercept in
//      (-pi, pi]; recentred once when |t0_corr| > 2 / band (_param_est,
//      :124-153);
//   4. the envelope: |V| / (2 pi f) symmetrised about f0 (_get_sym_amps,
//      :357-375), the phase's odd-polynomial fit (get_ang_func, :239-260,
//      solved here as the linear least-squares problem curve_fit converges
//      to), inverse FFT rolled to the peak (calc_envelope, :377-429), and
//      its mean, width and skewness (get_mu/get_sig/get_skewness, :435-451).
// Transforms are direct sums in FP64 with exact integer phase reduction, one
// output bin per thread: term m of bin k takes entry k m mod N of a table of
// sincospi(2 r / N) in shared memory, the index advanced by an addition (a
// sincospi and two 64-bit remainders per term were most of its time).  The
// scans whose order matters (running sums, the phase unwrapping) stay on one
// thread, over terms that all threads form; searches, peaks and per-bin
// values run on all of them.
#include <climits>

#include "sj_internal.h"

namespace sj {

namespace {

constexpr int PH_THREADS = 128;
constexpr double PI = 3.141592653589793;
constexpr double CUT_ALPHA = 0.1;        // scripts/phases.py:24
constexpr double DIV_S = 4000.0;         // :17
constexpr int MAX_LOWPASS_EVALS = 4;     // :28
constexpr double NOISE_THRESH = 0.1;     // signal.__init__ default

struct Ctl {
    int t0_ind;         // current roll of the series
    int f0_ind;         // _est_f0's index
    int f_min, f_max;   // band [f_min, f_max)
    int go;             // loop control set by thread 0
    int noise, count, high;  // is_noisy: to be evaluated; peaks prominent enough; one above 3 f0
    double cent;        // centre of the next low-pass step, < 0: none
    int status;
    int lowpass_steps;
    double f0, low_stren, last_cent;
    double t0_corr, phi;
    double poly[4];     // p1, p3, p5, p7 of the phase fit
};

// Block-wide reduction of (value, index) pairs to the largest value's first
// index.  Every thread passes its best candidate (idx = INT_MAX: none).
template <typename Greater>
__device__ int block_first(double v, double w, int idx, Greater greater) {
    __shared__ double sv[PH_THREADS / 32], sw[PH_THREADS / 32];
    __shared__ int si[PH_THREADS / 32];
    auto take = [&](double v2, double w2, int i2) {
        if (i2 != INT_MAX && (idx == INT_MAX || greater(v2, w2, v, w) || (!greater(v, w, v2, w2) && i2 < idx)))
            v = v2, w = w2, idx = i2;
    };
    for (int o = 16; o > 0; o >>= 1) {
        const double v2 = __shfl_down_sync(0xffffffffu, v, o), w2 = __shfl_down_sync(0xffffffffu, w, o);
        const int i2 = __shfl_down_sync(0xffffffffu, idx, o);
        take(v2, w2, i2);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sv[threadIdx.x >> 5] = v, sw[threadIdx.x >> 5] = w, si[threadIdx.x >> 5] = idx;
    __syncthreads();
    v = sv[0], w = sw[0], idx = si[0];
    for (int q = 1; q < PH_THREADS / 32; ++q) take(sv[q], sw[q], si[q]);
    return idx;
}

// numpy's argmax: the first index of the largest value (0 when the first is
// not a number, which nothing exceeds); f(i) the values
template <typename F>
__device__ int argmax(int n, F f) {
    double best = 0.0;
    int at = INT_MAX;
    for (int i = threadIdx.x; i < n; i += PH_THREADS) {
        const double x = f(i);
        if (!isnan(x) && (at == INT_MAX || x > best)) best = x, at = i;
    }
    const int r = block_first(best, 0.0, at, [](double a, double, double b, double) { return a > b; });
    return r == INT_MAX || isnan(f(0)) ? 0 : r;
}

// fix_angle (scripts/phases.py:51-61)
__device__ double fix_angle(double theta) {
    if (theta > PI) {
        theta -= 2 * PI * floor(theta / (2 * PI));
        if (theta > PI) theta -= 2 * PI;
    } else if (theta <= -PI) {
        theta += 2 * PI * (floor(-theta / (2 * PI)) + 1);
        if (theta > PI) theta -= 2 * PI;
    }
    return theta;
}

// fix_angle_seq (:63-74) in place: each angle moved by 2 pi when that brings
// it closer to the one before (the shift carries to every later angle)
__device__ void fix_angle_seq(double* a, int n) {
    for (int i = 1; i < n; ++i) {
        const double d = fabs(a[i] - a[i - 1]);
        double s = 0.0;
        if (fabs(a[i] + 2 * PI - a[i - 1]) < d)
            s = 2 * PI;
        else if (fabs(a[i] - 2 * PI - a[i - 1]) < d)
            s = -2 * PI;
        if (s != 0.0)
            for (int j = i; j < n; ++j) a[j] += s;
    }
}

// scipy.signal.find_peaks without conditions: local maxima, a flat top
// counted once at its middle (left of centre for an even width); the first
// and last samples are never peaks.  The peak whose rise ends at i (-1: none),
// each i by itself.
__device__ int peak_from(const double* x, int n, int i) {
    const int i_max = n - 1;
    if (i < 1 || i >= i_max || !(x[i - 1] < x[i])) return -1;
    int ahead = i + 1;
    while (ahead < i_max && x[ahead] == x[i]) ++ahead;
    return x[ahead] < x[i] ? (i + ahead - 1) / 2 : -1;
}

// scipy.signal.peak_prominences with no window
__device__ double prominence(const double* x, int n, int peak) {
    double left_min = x[peak];
    for (int i = peak; i >= 0 && x[i] <= x[peak]; --i)
        if (x[i] < left_min) left_min = x[i];
    double right_min = x[peak];
    for (int i = peak; i <= n - 1 && x[i] <= x[peak]; ++i)
        if (x[i] < right_min) right_min = x[i];
    return x[peak] - fmax(left_min, right_min);
}

__device__ __forceinline__ int pmod(long long a, int m) {
    const long long r = a % m;
    return (int)(r < 0 ? r + m : r);
}

// tab[r] = (cos, sin)(2 pi r / N)
__device__ void phase_table(double2* tab, int N) {
    for (int r = threadIdx.x; r < N; r += PH_THREADS) {
        double s, c;
        sincospi(2.0 * (double)r / (double)N, &s, &c);
        tab[r] = make_double2(c, s);
    }
}

// out[k] = 2 sum_m v[(m + shift) mod N] e^{-i 2 pi k m / N}, k < M (2 rfft of
// the rolled series), one bin per thread; x: the rolled series in shared memory
__device__ void rfft2_rolled(const double* v, int N, int M, int shift, const double2* tab, double* x, double2* out) {
    const int s0 = pmod(shift, N);
    for (int m = threadIdx.x; m < N; m += PH_THREADS) x[m] = v[m + s0 < N ? m + s0 : m + s0 - N];
    __syncthreads();
    for (int k = threadIdx.x; k < M; k += PH_THREADS) {
        double re = 0.0, im = 0.0;
        int r = 0;
        for (int m = 0; m < N; ++m) {
            const double2 e = tab[r];
            re += x[m] * e.x;
            im -= x[m] * e.y;
            r += k;
            if (r >= N) r -= N;
        }
        out[k] = make_double2(2.0 * re, 2.0 * im);
    }
    __syncthreads();
}

// _apply_lowpass (:278-284): vf = vf0 sinc((f - cent) strength) ...
__device__ void lowpass_spectrum(const double2* vf0, int M, double df, double cent, double strength, double2* vf,
                                 double* mags) {
    for (int k = threadIdx.x; k < M; k += PH_THREADS) {
        const double x = ((double)k * df - cent) * strength;
        const double y = PI * (x == 0.0 ? 1.0e-20 : x);
        const double s = sin(y) / y;
        const double2 a = vf0[k];
        vf[k] = make_double2(a.x * s, a.y * s);
        mags[k] = hypot(a.x * s, a.y * s);
    }
    __syncthreads();
}
// ... and v = the inverse real FFT (length L = 2 (M - 1)) rolled by t0,
// zero-padded to N (only the last low-pass step's is used); sh: vf's copy
__device__ void lowpass_series(const double2* vf, int N, int M, int t0, const double2* tabL, double2* sh, double* v) {
    const int L = 2 * (M - 1);
    for (int k = threadIdx.x; k < M; k += PH_THREADS) sh[k] = vf[k];
    __syncthreads();
    for (int n = threadIdx.x; n < N; n += PH_THREADS) {
        if (n >= L) {
            v[n] = 0.0;
            continue;
        }
        const int m = pmod((long long)n - t0, L);
        // x[m] = (Re X0 + Re X_{L/2} (-1)^m + 2 sum_{0<k<L/2} Re(X_k e^{i 2 pi k m / L})) / L
        double acc = sh[0].x + ((m & 1) ? -sh[M - 1].x : sh[M - 1].x);
        int r = m;
        for (int k = 1; k < M - 1; ++k) {
            const double2 e = tabL[r];
            acc += 2.0 * (sh[k].x * e.x - sh[k].y * e.y);
            r += m;
            if (r >= L) r -= L;
        }
        v[n] = acc / (double)L;
    }
    __syncthreads();
}

// _get_freq_fwhm (:107-122): the farthest bin above the cut on each side of f0
__device__ void freq_band(const double* mags, int M, int f0i, double threshold, Ctl& C) {
    __syncthreads();
    if (threadIdx.x == 0) C.f_min = C.f_max = f0i;
    __syncthreads();
    const double cut = mags[f0i] * threshold;
    const int jb = min(f0i, M - f0i - 1);
    for (int j = threadIdx.x; j < jb; j += PH_THREADS) {
        if (mags[f0i - j] > cut) atomicMin(&C.f_min, f0i - j - 1);
        if (mags[f0i + j] > cut) atomicMax(&C.f_max, f0i + j + 1);
    }
    __syncthreads();
}

// linregress of the unwrapped band phase ang (in place) against frequency (thread 0)
__device__ void band_regression(int lo, int hi, double df, double* ang, double* slope, double* intercept) {
    const int n = hi - lo;
    fix_angle_seq(ang, n);
    double xm = 0.0, ym = 0.0;
    for (int i = 0; i < n; ++i) xm += (double)(lo + i) * df, ym += ang[i];
    xm /= n;
    ym /= n;
    double sxx = 0.0, sxy = 0.0;
    for (int i = 0; i < n; ++i) {
        const double dx = (double)(lo + i) * df - xm;
        sxx += dx * dx;
        sxy += dx * (ang[i] - ym);
    }
    *slope = sxy / sxx;
    *intercept = ym - *slope * xm;
}

// u^k correctly rounded (double-double product, then one rounding), as the
// reference's numpy power gives it
__device__ double pow_int(double u, int k) {
    double hi = u, lo = 0.0;
    for (int i = 1; i < k; ++i) {
        const double p = __dmul_rn(hi, u);
        const double e = fma(hi, u, -p);                    // hi * u - p exactly
        const double l = __dadd_rn(__dmul_rn(lo, u), e);
        const double h2 = __dadd_rn(p, l);
        lo = __dadd_rn(l, -__dsub_rn(h2, p));
        hi = h2;
    }
    return hi;
}

// The phase model p7 u^7 + p5 u^5 + p3 u^3 + p1 u + p0, summed left to right
// without contraction, as the reference's lambda evaluates it.
__device__ double odd_model(const double* q, double u, double u3, double u5, double u7) {
    double m = __dmul_rn(q[4], u7);
    m = __dadd_rn(m, __dmul_rn(q[3], u5));
    m = __dadd_rn(m, __dmul_rn(q[2], u3));
    m = __dadd_rn(m, __dmul_rn(q[1], u));
    return __dadd_rn(m, q[0]);
}

// Least squares of angles ~ p0 + p1 u + p3 u^3 + p5 u^5 + p7 u^7, u = f - f0,
// by Householder QR; a: 5 n doubles, b: n doubles (shared memory).  curve_fit
// starts from p = 1 and takes forward differences with step 2^-26 |p_j|
// (MINPACK's fdjac2); a parameter whose difference column is zero in every
// band bin (its term is lost to rounding) never moves from 1, so it is held
// at 1 here and the others are fitted to what remains.  The rows are formed by
// all threads; warp 0 reduces, one lane per column (each column's sums in
// row order).
__device__ void odd_poly_fit(const double* ang, int lo, int n, double df, double f0, double* a, double* b,
                             double* poly) {
    constexpr int P = 5;
    __shared__ int moves[P];
    const double h = 1.4901161193847656e-08;  // sqrt(DBL_EPSILON)
    if (threadIdx.x < P) moves[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += PH_THREADS) {
        const double u = (double)(lo + i) * df - f0;
        const double u3 = pow_int(u, 3), u5 = pow_int(u, 5), u7 = pow_int(u, 7);
        const double one[P] = {1.0, 1.0, 1.0, 1.0, 1.0};
        const double m1 = odd_model(one, u, u3, u5, u7);
        for (int j = 0; j < P; ++j) {
            double q[P] = {1.0, 1.0, 1.0, 1.0, 1.0};
            q[j] = 1.0 + h;
            if (!(odd_model(q, u, u3, u5, u7) == m1)) moves[j] = 1;
        }
    }
    __syncthreads();
    int free_idx[P], nf = 0;
    for (int j = 0; j < P; ++j)
        if (moves[j]) free_idx[nf++] = j;
    for (int i = threadIdx.x; i < n; i += PH_THREADS) {
        const double u = (double)(lo + i) * df - f0;
        const double col[P] = {1.0, u, pow_int(u, 3), pow_int(u, 5), pow_int(u, 7)};
        double y = ang[i];
        for (int j = 0; j < P; ++j)
            if (!moves[j]) y -= col[j];
        b[i] = y;
        for (int c = 0; c < nf; ++c) a[c * n + i] = col[free_idx[c]];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        for (int c = 0; c < nf; ++c) {
            double alpha = 0.0, v0 = 0.0, vtv = 0.0;
            if (lane == 0) {
                double nrm = 0.0;
                for (int i = c; i < n; ++i) nrm += a[c * n + i] * a[c * n + i];
                nrm = sqrt(nrm);
                alpha = a[c * n + c] > 0 ? -nrm : nrm;
                v0 = a[c * n + c] - alpha;
                // reflector v = (v0, a[c+1..]) with H = I - 2 v v^T / (v^T v)
                vtv = v0 * v0;
                for (int i = c + 1; i < n; ++i) vtv += a[c * n + i] * a[c * n + i];
            }
            v0 = __shfl_sync(0xffffffffu, v0, 0);
            vtv = __shfl_sync(0xffffffffu, vtv, 0);
            if (vtv == 0.0) continue;
            if (lane > c && lane <= nf) {  // the columns to the right, then the right-hand side
                double* x = lane == nf ? b : a + lane * n;
                double d = v0 * x[c];
                for (int i = c + 1; i < n; ++i) d += a[c * n + i] * x[i];
                const double f = 2.0 * d / vtv;
                x[c] -= f * v0;
                for (int i = c + 1; i < n; ++i) x[i] -= f * a[c * n + i];
            }
            __syncwarp();
            if (lane == 0) a[c * n + c] = alpha;
            __syncwarp();
        }
        if (lane == 0) {
            double pf[P];
            for (int c = nf - 1; c >= 0; --c) {
                double s = b[c];
                for (int cc = c + 1; cc < nf; ++cc) s -= a[cc * n + c] * pf[cc];
                pf[c] = s / a[c * n + c];
            }
            double p[P] = {1.0, 1.0, 1.0, 1.0, 1.0};
            for (int c = 0; c < nf; ++c) p[free_idx[c]] = pf[c];
            poly[0] = p[1];
            poly[1] = p[2];
            poly[2] = p[3];
            poly[3] = p[4];
        }
    }
    __syncthreads();
}

// sum of x[0 .. n) in order (one thread)
__device__ __forceinline__ double sum_in_order(const double* x, int n) {
    double s = 0.0;
    for (int i = 0; i < n; ++i) s += x[i];
    return s;
}

}  // namespace

// Per-series workspace layout, in doubles, for N samples (M = N / 2 + 1
// bins): every array starts on a 16-double (128-byte) boundary, so the
// double2 arrays are 16-byte aligned whatever N is.
struct PhaseLay {
    long long v0, v, vabs2, vf0, vf, mags, ef, vef, env, envt, total;
    __host__ __device__ explicit PhaseLay(int N) {
        const long long M = N / 2 + 1;
        auto al = [](long long x) { return (x + 15) & ~15LL; };
        v0 = 0;
        v = v0 + al(N);
        vabs2 = v + al(N);
        vf0 = vabs2 + al(N);
        vf = vf0 + al(2 * M);
        mags = vf + al(2 * M);
        ef = mags + al(M);
        vef = ef + al(N);
        env = vef + al(N);
        envt = env + al(2LL * N);
        total = envt + al(2LL * N);
    }
};
// Shared memory of a block: the phase table of N, that of L = 2 (M - 1) where
// it differs, and a buffer of N + 2 doubles.
static size_t phase_smem(int N) {
    const int L = 2 * (N / 2);
    return (2 * (size_t)N + (L == N ? 0 : 2 * (size_t)L) + N + 2) * sizeof(double);
}

// phase_smem of the longest series (4096 samples at most, odd ones need more)
constexpr int PH_MAX_SMEM = (2 * 4095 + 2 * 4094 + 4095 + 2) * (int)sizeof(double);

long long phase_workspace(int N) { return PhaseLay(N).total; }

// series q: v[q * s_series + k * s_sample], k < N; t[k] the sample times.
// 384 series of 200 samples: 4.26 ms before the phase table and the parallel
// scans, 0.30 ms with them (2.5 blocks per SM; about 0.1 ms is the FP64 pipe's
// share, the rest the ordered sums and the fit, chains of 62-cycle additions).
__global__ void __launch_bounds__(PH_THREADS)
k_phases(const double* __restrict__ vin, long long s_series, long long s_sample, int N, const double* __restrict__ t,
         double lowpass_inc, double* __restrict__ work, long long wstride, sj_phase_result* __restrict__ out) {
    extern __shared__ __align__(16) double dyn[];
    __shared__ Ctl C;
    __shared__ double ang[256], fit[6 * 256], part[2];
    __shared__ unsigned peaks[4096 / 32];
    const int q = blockIdx.x, tid = threadIdx.x;
    const int M = N / 2 + 1, LL = 2 * (M - 1);
    double2* const tab = reinterpret_cast<double2*>(dyn);
    double2* const tabL = LL == N ? tab : tab + N;
    double* const buf = reinterpret_cast<double*>(tabL + LL);  // N + 2 doubles
    const PhaseLay lay(N);
    double* w = work + (long long)q * wstride;  // wstride: a multiple of 16 doubles
    double* v0 = w + lay.v0;                    // original series
    double* v = w + lay.v;                      // v_pts
    double* vabs2 = w + lay.vabs2;              // v^2 (find_peaks input)
    double2* vf0 = reinterpret_cast<double2*>(w + lay.vf0);   // [M]
    double2* vf = reinterpret_cast<double2*>(w + lay.vf);     // [M]
    double* mags = w + lay.mags;                // [M]
    double* ef = w + lay.ef;                    // [N]
    double* vef = w + lay.vef;                  // [N]
    double2* env = reinterpret_cast<double2*>(w + lay.env);   // [N] Fourier envelope
    double2* envt = reinterpret_cast<double2*>(w + lay.envt); // [N] envelope
    const double dt = t[1] - t[0];
    const double df = 1.0 / ((double)N * dt);  // rfftfreq spacing

    for (int k = tid; k < N; k += PH_THREADS) {
        const double x = vin[(long long)q * s_series + (long long)k * s_sample];
        v0[k] = x;
        v[k] = x;
        vabs2[k] = x * x;
    }
    phase_table(tab, N);
    if (LL != N) phase_table(tabL, LL);
    __syncthreads();
    // _guess_t0_ind: the peaks of v^2, summed in order
    int* const pos = reinterpret_cast<int*>(buf);
    for (int i0 = 0; i0 < N; i0 += PH_THREADS) {
        const int i = i0 + tid, at = peak_from(vabs2, N, i);
        const unsigned m = __ballot_sync(0xffffffffu, at >= 0);
        if (i < N) pos[i] = at;
        if ((tid & 31) == 0 && i < N) peaks[i >> 5] = m;
    }
    __syncthreads();
    if (tid == 0) {
        double at = 0.0, tm = 0.0;
        for (int c = 0; c < (N + 31) / 32; ++c)
            for (unsigned m = peaks[c]; m; m &= m - 1) {
                const int i = pos[32 * c + __ffs(m) - 1];
                at += (double)i * fabs(v0[i]);
                tm += fabs(v0[i]);
            }
        C.t0_ind = tm <= 0.0 ? 0 : (int)(at / tm);
        C.status = 0;
        C.f0 = 0.0;
        C.f0_ind = 0;
        C.low_stren = 0.0;
        C.last_cent = 0.0;
        C.lowpass_steps = 0;
    }
    __syncthreads();
    rfft2_rolled(v, N, M, C.t0_ind, tab, buf, vf0);
    for (int k = tid; k < M; k += PH_THREADS) {
        vf[k] = vf0[k];
        mags[k] = hypot(vf0[k].x, vf0[k].y);
    }
    __syncthreads();
    // the low-pass loop of signal.__init__
    for (;;) {
        const int fi = argmax(M, [&](int i) { return mags[i]; });
        const int L = min(2 * fi, M);
        // the terms of numpy.trapz of |V| f and |V| below 2 fi, summed in order
        for (int i = tid; i + 1 < L; i += PH_THREADS) {
            buf[i] = (mags[i] * ((double)i * df) + mags[i + 1] * ((double)(i + 1) * df)) / 2.0;
            buf[M + i] = (mags[i] + mags[i + 1]) / 2.0;
        }
        __syncthreads();
        if (tid == 0) part[0] = sum_in_order(buf, max(0, L - 1));
        if (tid == 32) part[1] = sum_in_order(buf + M, max(0, L - 1));
        __syncthreads();
        if (tid == 0) {
            C.go = C.noise = C.count = C.high = 0;
            const double f0 = part[0] / part[1];
            const double r = rint(f0 / df);
            if (!isfinite(f0) || !(r < (double)M)) {
                C.status = SJ_PHASE_BAD_F0;
            } else {
                C.f0 = f0;
                C.f0_ind = (int)r;
                C.cent = -1.0;
                if (!(C.low_stren >= MAX_LOWPASS_EVALS * lowpass_inc)) {
                    if (C.f0_ind > M / 2)
                        C.cent = 0.0;
                    else
                        C.noise = 1;
                }
            }
        }
        __syncthreads();
        if (C.status) break;
        if (C.noise) {
            // is_noisy: two or more peaks of prominence >= 0.1 |V(f0)|, one above 3 f0
            const double pmin = NOISE_THRESH * mags[C.f0_ind];
            for (int i = tid; i < M; i += PH_THREADS) {
                const int at = peak_from(mags, M, i);
                if (at >= 0 && prominence(mags, M, at) >= pmin) {
                    atomicAdd(&C.count, 1);
                    if (at > 3 * C.f0_ind) C.high = 1;
                }
            }
            __syncthreads();
        }
        if (tid == 0) {
            if (C.noise && C.count >= 2 && C.high) C.cent = (double)C.f0_ind * df / 2.0;
            if (C.cent >= 0.0) {
                C.low_stren += lowpass_inc;
                C.last_cent = C.cent;
                C.lowpass_steps += 1;
                C.go = 1;
            }
        }
        __syncthreads();
        if (!C.go) break;
        lowpass_spectrum(vf0, M, df, C.last_cent, C.low_stren, vf, mags);
    }
    if (!C.status && C.lowpass_steps > 0) lowpass_series(vf, N, M, C.t0_ind, tabL, reinterpret_cast<double2*>(buf), v);
    // _param_est, recentred at most once
    // (the loop reads the control words only after a barrier: thread 0 writes
    // them at the top of a pass while the others wait)
    for (int pass = 0; pass < 2 && !C.status; ++pass) {
        freq_band(mags, M, C.f0_ind, CUT_ALPHA, C);
        const int lo = C.f_min, n = C.f_max - lo;
        if (n > 0 && n <= 256)
            for (int i = tid; i < n; i += PH_THREADS) ang[i] = atan2(vf[lo + i].y, vf[lo + i].x);
        __syncthreads();
        if (tid == 0) {
            C.go = 0;
            if (n == 0) {
                // the recentring test divides by the band width on every pass
                C.status = SJ_PHASE_EMPTY_BAND;
            } else if (n > 256) {
                C.status = SJ_PHASE_WIDE_BAND;
            } else {
                double slope, icpt;
                band_regression(lo, C.f_max, df, ang, &slope, &icpt);
                C.t0_corr = -slope / (2 * PI);
                C.phi = fix_angle(icpt);
                if (pass == 0 && fabs(C.t0_corr) > 2.0 / (double)n) {
                    C.t0_ind += (int)(C.t0_corr / dt);
                    C.go = 1;
                }
            }
        }
        __syncthreads();
        if (C.status || !C.go) break;
        rfft2_rolled(v, N, M, C.t0_ind, tab, buf, env);  // env as scratch for the rolled spectrum
        lowpass_spectrum(env, M, df, C.last_cent, C.low_stren, vf, mags);
        lowpass_series(vf, N, M, C.t0_ind, tabL, reinterpret_cast<double2*>(buf), v);
    }
    __syncthreads();
    // after a recentring, t_pts[t0_ind] must exist (Python indexing: -N <= t0_ind < N)
    if (tid == 0 && !C.status && (C.t0_ind >= N || C.t0_ind < -N)) C.status = SJ_PHASE_BAD_T0;
    __syncthreads();
    if (C.status) {
        if (tid == 0) {
            sj_phase_result r = {};
            r.f0 = C.f0;
            r.f0_ind = C.f0_ind;
            r.status = C.status;
            out[q] = r;
        }
        return;
    }
    // calc_envelope, symmetric mode: t0_ind = argmax |v_pts|
    const int best = argmax(N, [&](int i) { return fabs(v[i]); });
    const double f0 = C.f0;
    double* vec = reinterpret_cast<double*>(envt);  // |V| / (2 pi f + exp(-DIV_S f / f0))
    for (int i = tid; i < N; i += PH_THREADS) ef[i] = vef[i] = 0.0;
    for (int k = tid; k < M; k += PH_THREADS) {
        const double f = (double)k * df;
        vec[k] = mags[k] / (2 * PI * f + exp(-DIV_S * f / f0));
    }
    __syncthreads();
    const int fi = (int)(f0 / df);
    const double lrp = f0 - fi * df;
    const int nn = min(fi, M - fi - 1);
    for (int i = tid; i < nn; i += PH_THREADS) {
        const double a = 0.5 * (vec[fi - i + 1] - vec[fi - i] + vec[fi + i + 1] - vec[fi + i]) * lrp / df +
                         0.5 * (vec[fi - i] + vec[fi + i]);
        const int ni = i == 0 ? 0 : N - i;
        if (i != 0) {
            vef[ni] = a;
            ef[ni] = 2 * PI * (f0 - (double)i * df) * a;
        }
        vef[i] = a;
        ef[i] = 2 * PI * (f0 + (double)i * df) * a;
    }
    // get_ang_func: the phase in the band (unwrapped by the regression) fitted by an odd polynomial + constant
    const int n_band = C.f_max - C.f_min;
    if (tid == 0) {
        C.t0_ind = best;
        C.go = 0;
        if (n_band < 5 || n_band > 256) C.status = n_band < 5 ? SJ_PHASE_NARROW_BAND : SJ_PHASE_WIDE_BAND;
    }
    __syncthreads();
    if (C.status) {
        if (tid == 0) {
            sj_phase_result r = {};
            r.f0 = C.f0;
            r.phi = C.phi;
            r.t0_corr = C.t0_corr;
            r.f0_ind = C.f0_ind;
            r.band_lo = C.f_min;
            r.band_hi = C.f_max;
            r.lowpass_steps = C.lowpass_steps;
            r.status = C.status;
            out[q] = r;
        }
        return;
    }
    odd_poly_fit(ang, C.f_min, n_band, df, f0, fit, fit + 5 * 256, C.poly);
    // env_fourier = ef e^{i vp(fftfreq)}, envelope = 2 roll(ifft(env_fourier), t0)
    for (int k = tid; k < N; k += PH_THREADS) {
        const int kk = k < (N + 1) / 2 ? k : k - N;  // fftfreq order
        const double x = (double)kk * df;
        const double x2 = x * x;
        const double ph = C.poly[3] * (x2 * x2 * x2 * x) + C.poly[2] * (x2 * x2 * x) + C.poly[1] * (x2 * x) +
                          C.poly[0] * x;
        double s, c;
        sincos(ph, &s, &c);
        const double2 e = make_double2(ef[k] * c, ef[k] * s);
        env[k] = e;
        if (k >= nn && k <= N - nn && (e.x != 0.0 || e.y != 0.0)) C.go = 1;
    }
    __syncthreads();
    // ef is 0 from nn to N - nn: those terms add 0 (unless the phase is not finite there, C.go)
    const int k1 = C.go ? N : max(nn, 0), k2 = C.go ? N : N - max(nn, 1) + 1;
    for (int n = tid; n < N; n += PH_THREADS) {
        const int m = pmod((long long)n - best, N);
        double re = 0.0, im = 0.0;
        auto terms = [&](int ka, int kb) {
            int r = (int)(((long long)ka * m) % N);
            for (int k = ka; k < kb; ++k) {
                const double2 e = tab[r], x = env[k];
                re += x.x * e.x - x.y * e.y;
                im += x.x * e.y + x.y * e.x;
                r += m;
                if (r >= N) r -= N;
            }
        };
        terms(0, k1);
        terms(k2, N);
        envt[n] = make_double2(2.0 * re / N, 2.0 * im / N);
    }
    __syncthreads();
    // get_skewness on |envelope| normalised to unit area: numpy.trapz' terms formed by all threads, summed in order
    double* a = ef;       // |env|, then normalised
    double* y2 = vabs2;
    double* const buf2 = reinterpret_cast<double*>(tab);  // the table is done with
    for (int i = tid; i < N; i += PH_THREADS) a[i] = hypot(envt[i].x, envt[i].y);
    __syncthreads();
    for (int i = tid; i + 1 < N; i += PH_THREADS) buf[i] = (a[i] + a[i + 1]) / 2.0;
    __syncthreads();
    if (tid == 0) part[0] = sum_in_order(buf, N - 1) * dt;
    __syncthreads();
    const double area = part[0];
    for (int i = tid; i < N; i += PH_THREADS) {
        a[i] = a[i] / area;
        vef[i] = a[i] * t[i];
    }
    __syncthreads();
    for (int i = tid; i + 1 < N; i += PH_THREADS) buf[i] = (vef[i] + vef[i + 1]) / 2.0;
    __syncthreads();
    if (tid == 0) part[0] = sum_in_order(buf, N - 1) * dt;
    __syncthreads();
    const double mu = part[0];
    for (int i = tid; i < N; i += PH_THREADS) {
        const double d = t[i] - mu;
        vef[i] = a[i] * ((t[i] - mu) * (t[i] - mu));
        y2[i] = a[i] * (d * d * d);
    }
    __syncthreads();
    for (int i = tid; i + 1 < N; i += PH_THREADS) {
        buf[i] = (vef[i] + vef[i + 1]) / 2.0;
        buf2[i] = (y2[i] + y2[i + 1]) / 2.0;
    }
    __syncthreads();
    if (tid == 0) part[0] = sum_in_order(buf, N - 1);
    if (tid == 32) part[1] = sum_in_order(buf2, N - 1);
    __syncthreads();
    // numpy's argmax of a complex array: largest real part, then imaginary
    double bx = 0.0, by = 0.0;
    int at = INT_MAX;
    for (int i = tid; i < N; i += PH_THREADS) {
        const double2 e = envt[i];
        if (!isnan(e.x) && (at == INT_MAX || e.x > bx || (e.x == bx && e.y > by))) bx = e.x, by = e.y, at = i;
    }
    int k = block_first(bx, by, at, [](double x, double y, double x2, double y2_) { return x > x2 || (x == x2 && y > y2_); });
    if (k == INT_MAX || isnan(envt[0].x)) k = 0;
    if (tid == 0) {
        const double sig = sqrt(part[0] * dt);
        const double skew = part[1] / (sig * sig * sig);
        sj_phase_result r = {};
        r.f0 = C.f0;
        r.phi = C.phi;
        r.t0_corr = C.t0_corr;
        r.t0 = t[best];
        r.amp[0] = envt[k].x;
        r.amp[1] = envt[k].y;
        r.mu = mu;
        r.sig = sig;
        r.skew = skew;
        r.f0_ind = C.f0_ind;
        r.band_lo = C.f_min;
        r.band_hi = C.f_max;
        r.lowpass_steps = C.lowpass_steps;
        r.status = 0;
        out[q] = r;
    }
}

cudaError_t launch_phases(const double* d_v, long long s_series, long long s_sample, int n_series, int N,
                          const double* d_t, double lowpass_inc, double* d_work, sj_phase_result* d_out,
                          cudaStream_t s) {
    if (n_series <= 0) return cudaSuccess;
    const size_t smem = phase_smem(N);
    if (smem > 32 * 1024) {
        // the attribute is the process's: always the largest size, so that callers of
        // several threads do not set each other's
        cudaError_t e = cudaFuncSetAttribute(k_phases, cudaFuncAttributeMaxDynamicSharedMemorySize, PH_MAX_SMEM);
        if (e != cudaSuccess) return e;
    }
    k_phases<<<n_series, PH_THREADS, smem, s>>>(d_v, s_series, s_sample, N, d_t, lowpass_inc, d_work,
                                             phase_workspace(N), d_out);
    return cudaGetLastError();
}

}  // namespace sj
