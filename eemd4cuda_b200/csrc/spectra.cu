// spectra.cu -- the IMF spectra stage on the device (sm_100a): Hilbert
// instantaneous frequency / amplitude and the STFT of batched float64 rows.
//
// Hilbert:  the row's Hilbert transform through real transforms (k_hil_small,
//           or k_hil_cols, k_hil_rows, k_hil_cols), then k_hil_out (phase
//           differences wrapped as np.unwrap does, centred differences as
//           np.gradient does, |z|).  The frequency needs only neighbouring
//           phase differences, so no scan over the unwrapped phase is formed.
//           Rows beyond the plan's length: k_promote (complex rows) -> FFT ->
//           k_analytic (weights 1 / 2 / 0 on DC (and Nyquist) / positive /
//           negative frequencies, 1/N) -> inverse FFT -> k_if_amp.
// STFT:     k_stft in one launch (frames of up to 4096 samples with factors up
//           to 31); else x -> k_frames (zero-extended by nperseg/2 at
//           both ends, periodic Hann window, complex rows) -> FFT batched over
//           rows x frames -> k_stft_out (one-sided half, transposed to [F][T],
//           divided by the window sum).
// The FFTs are this file's own (below): no FFT library is linked.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "../../include/eemd_spectra.h"

namespace sp {

constexpr double PI = 3.141592653589793238462643383279502884;

// analytic spectrum from the full one: z[k] = w_k X[k] / N with w = 1 at DC
// (and at N/2 for even N), 2 on 1 <= k < N/2 (k < (N+1)/2 for odd N), 0 above
__global__ void k_analytic(const double2* __restrict__ spec, double2* out, int M, int64_t N) {
    const int64_t total = (int64_t)M * N;
    const double inv = 1.0 / (double)N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = i % N;
        double w;
        if (k == 0) w = 1.0;
        else if ((N & 1) == 0 && k == N / 2) w = 1.0;
        else if (2 * k < N) w = 2.0;
        else w = 0.0;
        double2 z = make_double2(0.0, 0.0);
        if (w != 0.0) {
            const double2 X = spec[i];
            z = make_double2(X.x * w * inv, X.y * w * inv);
        }
        out[i] = z;
    }
}

// complex rows from real ones
__global__ void k_promote(const double* __restrict__ x, double2* z, int64_t total) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x)
        z[i] = make_double2(x[i], 0.0);
}

// the unwrapped difference of two wrapped phases (np.unwrap, period 2 pi,
// discont pi): dd itself when |dd| < pi, else dd taken into [-pi, pi) with
// -pi mapped to pi when dd > 0.  A difference of two wrapped phases is at most
// 2 pi, so numpy's floor-mod of dd + pi by 2 pi is one exact subtraction or one
// addition (its general form by fmod was half of the closing kernel's time:
// nearly every warp holds a sample that wraps).
__device__ __forceinline__ double unwrap_diff(double dd) {
    if (fabs(dd) < PI) return dd;
    const double a = dd + PI, b = 2.0 * PI;
    const double r = a >= b ? a - b : (a < 0.0 ? a + b : a);
    double d = r - PI;
    if (d == -PI && dd > 0.0) d = PI;
    return d;
}

__global__ void k_if_amp(const double2* __restrict__ z, double* inst_freq, double* inst_amp, int M, int64_t N,
                         double sr) {
    const int64_t total = (int64_t)M * N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i % N;
        const double2 c = z[i];
        const double p = atan2(c.y, c.x);
        double f;
        if (n == 0) {
            const double2 r = z[i + 1];
            f = unwrap_diff(atan2(r.y, r.x) - p) * sr;
        } else if (n == N - 1) {
            const double2 l = z[i - 1];
            f = unwrap_diff(p - atan2(l.y, l.x)) * sr;
        } else {
            const double2 l = z[i - 1], r = z[i + 1];
            f = (unwrap_diff(p - atan2(l.y, l.x)) + unwrap_diff(atan2(r.y, r.x) - p)) * sr * 0.5;
        }
        inst_freq[i] = f / (2.0 * PI);
        inst_amp[i] = hypot(c.x, c.y);
    }
}

// frames[m][j][n] = w[n] * x[m][j*step + n - half] (zero outside the row), complex
__global__ void k_frames(const double* __restrict__ x, double2* frames, int M, int64_t N, int nperseg, int step,
                         int T) {
    const int half = nperseg / 2;
    const int64_t total = (int64_t)M * T * nperseg;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int n = (int)(i % nperseg);
        const int64_t mj = i / nperseg;
        const int j = (int)(mj % T);
        const int64_t m = mj / T;
        const int64_t s = (int64_t)j * step + n - half;
        const double w = 0.5 - 0.5 * cos(2.0 * PI * (double)n / (double)nperseg);
        frames[i] = make_double2((s >= 0 && s < N) ? x[m * N + s] * w : 0.0, 0.0);
    }
}

// Z[m][f][t] = spec[m][t][f] / wsum (f < F of each frame's nperseg bins)
__global__ void k_stft_out(const double2* __restrict__ spec, double2* Z, int M, int F, int T, int nperseg,
                           double inv_wsum) {
    const int64_t total = (int64_t)M * F * T;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int t = (int)(i % T);
        const int64_t mf = i / T;
        const int f = (int)(mf % F);
        const int64_t m = mf / F;
        const double2 v = spec[(m * T + t) * nperseg + f];
        Z[i] = make_double2(v.x * inv_wsum, v.y * inv_wsum);
    }
}

size_t al(size_t b) { return (b + 255) / 256 * 256; }

unsigned grid_for(int64_t total) {
    const int64_t b = (total + 255) / 256;
    return (unsigned)(b < 148 * 32 ? (b > 0 ? b : 1) : 148 * 32);
}

// ---------------------------------------------------------------------------
// Complex FFT of batched rows, this library's own (no FFT library):
// Stockham autosort passes of radix 4, 2, 3, 5 (in shared memory 16 and 8 too)
// and of the odd primes up to 31
// (the formulation of Govindaraju et al., "High performance discrete Fourier
// transforms on graphics processors", SC'08: pass s reads x[j + q N/R],
// multiplies by the twiddle w^(q k) of the current sub-transform length
// Ns R (k = j mod Ns), takes a radix-R DFT and writes the results sorted, so
// no bit reversal is needed); a length with a prime factor above 31 goes
// through Bluestein's chirp-z identity, n k = (n^2 + k^2 - (k-n)^2) / 2, as a
// circular convolution of power-of-two length.  Unnormalised; sign -1 is the
// forward transform X[k] = sum_n x[n] exp(-2 pi i n k / N) (numpy's and
// scipy's), +1 the inverse.  Twiddles and chirps are formed on the fly with
// sincospi of an exactly reduced argument.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// i * sign * z
__device__ __forceinline__ double2 cisg(double2 z, int sign) {
    return sign < 0 ? make_double2(z.y, -z.x) : make_double2(-z.y, z.x);
}
// exp(sign 2 pi i num / den), num reduced exactly into [0, den)
__device__ __forceinline__ double2 twiddle(int64_t num, int64_t den, int sign) {
    int64_t r = num % den;
    if (r < 0) r += den;
    double s, c;
    sincospi(2.0 * ((double)r / (double)den), &s, &c);
    return make_double2(c, sign < 0 ? -s : s);
}

template <int R>
__device__ __forceinline__ void dft_small(double2 (&a)[R], int sign) {
    if constexpr (R == 8 || R == 16) {
        // R = 4 H points n = H n1 + n2, k = k1 + 4 k2: H radix-4 transforms, the
        // twiddles w_R^(n2 k1), 4 radix-H transforms
        constexpr int H = R / 4;
        // cos(pi m / 8), sin(pi m / 8)
        constexpr double c8[10] = {1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                                   -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613, -1.0,
                                   -0.92387953251128675613};
        constexpr double s8[10] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0,
                                   0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                                   -0.38268343236508977173};
        double2 b[H][4];
#pragma unroll
        for (int n2 = 0; n2 < H; ++n2) {
#pragma unroll
            for (int n1 = 0; n1 < 4; ++n1) b[n2][n1] = a[H * n1 + n2];
            dft_small<4>(b[n2], sign);
#pragma unroll
            for (int k1 = 1; k1 < 4; ++k1) {
                if (n2 == 0) continue;
                const int m = n2 * k1 * (16 / R);
                b[n2][k1] = cmul(b[n2][k1], make_double2(c8[m], sign < 0 ? -s8[m] : s8[m]));
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            double2 c[H];
#pragma unroll
            for (int n2 = 0; n2 < H; ++n2) c[n2] = b[n2][k1];
            dft_small<H>(c, sign);
#pragma unroll
            for (int k2 = 0; k2 < H; ++k2) a[k1 + 4 * k2] = c[k2];
        }
    } else if constexpr (R == 2) {
        const double2 t = a[1];
        a[1] = csub(a[0], t);
        a[0] = cadd(a[0], t);
    } else if constexpr (R == 3) {
        // w = exp(sign 2 pi i / 3) = -1/2 + sign i sqrt(3)/2
        const double h = 0.86602540378443864676;  // sqrt(3) / 2
        const double2 t1 = cadd(a[1], a[2]), t2 = csub(a[1], a[2]);
        const double2 m = make_double2(fma(-0.5, t1.x, a[0].x), fma(-0.5, t1.y, a[0].y));
        const double2 r = cisg(make_double2(h * t2.x, h * t2.y), sign);
        a[0] = cadd(a[0], t1);
        a[1] = cadd(m, r);
        a[2] = csub(m, r);
    } else if constexpr (R == 4) {
        const double2 t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
        const double2 t2 = cadd(a[1], a[3]), t3 = cisg(csub(a[1], a[3]), sign);
        a[0] = cadd(t0, t2);
        a[2] = csub(t0, t2);
        a[1] = cadd(t1, t3);
        a[3] = csub(t1, t3);
    } else if constexpr (R == 5) {
        // cos and sin of 2 pi / 5 and 4 pi / 5 from their closed forms
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
        const double2 t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]);
        const double2 t3 = csub(a[1], a[4]), t4 = csub(a[2], a[3]);
        const double2 m1 = make_double2(a[0].x + c1 * t1.x + c2 * t2.x, a[0].y + c1 * t1.y + c2 * t2.y);
        const double2 m2 = make_double2(a[0].x + c2 * t1.x + c1 * t2.x, a[0].y + c2 * t1.y + c1 * t2.y);
        const double2 r1 = cisg(make_double2(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y), sign);
        const double2 r2 = cisg(make_double2(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y), sign);
        a[0] = cadd(a[0], cadd(t1, t2));
        a[1] = cadd(m1, r1);
        a[4] = csub(m1, r1);
        a[2] = cadd(m2, r2);
        a[3] = csub(m2, r2);
    }
}

// butterfly j of a Stockham pass of radix R over one row of N (nb = N / R):
// reads x[j + q nb], twiddles by w^(q k) of the sub-transform length Ns R
// (k = j mod Ns), takes the radix-R DFT and writes y[(j / Ns) Ns R + k + q Ns]
template <int R>
__device__ __forceinline__ void bfly(const double2* x, double2* y, int64_t j, int64_t nb, int64_t Ns, int sign) {
    const int64_t k = j % Ns;
    double2 a[R];
#pragma unroll
    for (int q = 0; q < R; ++q) a[q] = x[j + q * nb];
    if (Ns > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) a[q] = cmul(a[q], twiddle((int64_t)q * k, Ns * R, sign));
    }
    dft_small<R>(a, sign);
    const int64_t base = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) y[base + q * Ns] = a[q];
}

// the same butterfly for an odd prime radix r <= 31 (a direct DFT of the r points)
__device__ __forceinline__ void bfly_prime(const double2* x, double2* y, int64_t j, int64_t nb, int64_t Ns, int r,
                                           int sign) {
    const int64_t k = j % Ns;
    double2 a[31];
    for (int q = 0; q < r; ++q) {
        a[q] = x[j + q * nb];
        if (q > 0 && Ns > 1) a[q] = cmul(a[q], twiddle((int64_t)q * k, Ns * r, sign));
    }
    const int64_t base = (j / Ns) * Ns * r + k;
    for (int q = 0; q < r; ++q) {
        double2 s = a[0];
        for (int p = 1; p < r; ++p) s = cadd(s, cmul(a[p], twiddle((int64_t)p * q, r, sign)));
        y[base + q * Ns] = s;
    }
}

// one Stockham pass of radix R over M rows of N: in -> out (distinct buffers)
template <int R>
__global__ void k_fft_pass(const double2* __restrict__ in, double2* __restrict__ out, int M, int64_t N, int64_t Ns,
                           int sign) {
    const int64_t nb = N / R;
    const int64_t total = (int64_t)M * nb;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = i / nb, j = i % nb;
        bfly<R>(in + m * N, out + m * N, j, nb, Ns, sign);
    }
}

__global__ void k_fft_pass_prime(const double2* __restrict__ in, double2* __restrict__ out, int M, int64_t N,
                                 int64_t Ns, int r, int sign) {
    const int64_t nb = N / r;
    const int64_t total = (int64_t)M * nb;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = i / nb, j = i % nb;
        bfly_prime(in + m * N, out + m * N, j, nb, Ns, r, sign);
    }
}

// ---------------------------------------------------------------------------
// Transforms in shared memory: every pass of a direct plan (no Bluestein) of
// length n <= SMEM_FFT_MAX over some rows of a CTA, in place, with a table of
// the twiddles made once per CTA.
//
// A pass is bound by latency (shared-memory loads, a few dependent float64
// operations, the barriers) and by the integer work per butterfly, so: radices
// up to 16 (4096 in three passes), 32-bit indices, quotients by a multiply with
// a per-pass reciprocal (the twiddle index q k (n / (Ns R)) is below n and needs
// no reduction at all), and one element of padding after every eight, which
// spreads the strided stores and table reads over the banks.  A thread holds
// up to 16 points in registers over the barrier between a pass's loads and its
// stores: one buffer instead of two, so that twice the CTAs share an SM and
// cover each other's barriers and global loads.
// ---------------------------------------------------------------------------
constexpr int SMEM_FFT_MAX = 4096;
constexpr int SMEM_FFT_MAXRAD = 16;  // factors of n <= 4096 (at most 12)
constexpr int FFT_THREADS = 512;     // at most
// Points per thread, P: 16 where many CTAs follow one another on an SM (fewer
// threads per transform, so more transforms at a time: the STFT of 11 rows of
// 480 000, 4096-sample frames, 100 against 118 us with 8), 8 where one wave of
// CTAs is all there is and its latency counts (Hilbert of 8 rows of 48 000: 46
// against 58 us with 16).  A pass of radix r takes whole butterflies of them.
__host__ __device__ constexpr int pass_points(int r, int P) { return r <= P ? r * (P / r) : r; }

struct SmemPlan {
    int n, nrad;
    int rad[SMEM_FFT_MAXRAD];
};

// The kernels of one call follow one another with programmatic dependent
// launches: each makes its tables while the one before drains, then waits for
// it here before the first access to what it wrote (or to what its own writes
// would overwrite).
// (A kernel's life then overlaps that kernel's writes: no const __restrict__
// pointers and no __ldg here, whose loads presume memory that stays unchanged.)
__device__ __forceinline__ void after_previous_kernel() {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// position of element i in a padded row, and the padded length of a row of n
__host__ __device__ __forceinline__ int pad8(int i) { return i + (i >> 3); }

// quotients by d >= 1 of dividends below 2^20 (i < 2^20, d <= 2^12: the
// reciprocal's error times i stays below 2^32)
struct Div {
    uint32_t m;
    __device__ __forceinline__ explicit Div(int d) : m(d > 1 ? 0xffffffffu / (uint32_t)d + 1u : 0u) {}
    __device__ __forceinline__ int operator()(int i) const { return m ? (int)__umulhi((uint32_t)i, m) : i; }
};

// tab[pad8(m)] = exp(2 pi i m / n), or with HALF exp(pi i m / n), m < n
template <bool HALF>
__device__ __forceinline__ void make_table(double2* tab, int n) {
    for (int m = threadIdx.x; m < n; m += blockDim.x) {
        double sv, cv;
        sincospi((HALF ? 1.0 : 2.0) * ((double)m / (double)n), &sv, &cv);
        tab[pad8(m)] = make_double2(cv, sv);
    }
}

// exp(sign 2 pi i m / n), m < n
template <bool HALF>
__device__ __forceinline__ double2 table_at(const double2* tab, int n, int m, int sign) {
    double2 v;
    if (HALF) {
        const bool far = 2 * m >= n;  // beyond half a turn: the negative of the entry half a turn back
        v = tab[pad8(far ? 2 * m - n : 2 * m)];
        if (far) v = make_double2(-v.x, -v.y);
    } else {
        v = tab[pad8(m)];
    }
    return make_double2(v.x, sign < 0 ? -v.y : v.y);
}

template <int R, bool HALF, int P>
__device__ __forceinline__ void smem_pass(double2* buf, const double2* tab, int n, int Ns, int sign, int rows, int ld) {
    constexpr int B = pass_points(R, P) / R;  // butterflies per thread
    const int nb = n / R, step = n / (Ns * R), total = rows * nb;
    const Div by_nb(nb), by_ns(Ns);
    double2 a[B][R];
    int at[B];  // first output
#pragma unroll
    for (int u = 0; u < B; ++u) {
        const int i = min((int)(threadIdx.x + u * blockDim.x), total - 1);  // (spare threads repeat the last one)
        const int row = rows > 1 ? by_nb(i) : 0, j = i - row * nb;
        const int jq = by_ns(j), k = j - jq * Ns;
        const double2* x = buf + row * ld;
#pragma unroll
        for (int q = 0; q < R; ++q) a[u][q] = x[pad8(j + q * nb)];
        if (Ns > 1) {
#pragma unroll
            for (int q = 1; q < R; ++q) a[u][q] = cmul(a[u][q], table_at<HALF>(tab, n, q * k * step, sign));
        }
        dft_small<R>(a[u], sign);
        at[u] = row * ld;
        // (row offset and position kept apart: padding applies within the row)
        at[u] |= (jq * Ns * R + k) << 16;
        asm volatile("" ::: "memory");  // one butterfly after the other: no loads drawn ahead
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < B; ++u) {
        if ((int)(threadIdx.x + u * blockDim.x) >= total) continue;
        double2* y = buf + (at[u] & 0xffff);
        const int base = at[u] >> 16;
#pragma unroll
        for (int q = 0; q < R; ++q) y[pad8(base + q * Ns)] = a[u][q];
    }
    __syncthreads();
}

// an odd prime radix 7 <= r <= 31: a direct DFT of the r points
template <bool HALF, int P>
__device__ __noinline__ void smem_pass_prime(double2* buf, const double2* tab, int n, int Ns, int r, int sign, int rows,
                                             int ld) {
    const int nb = n / r, step = n / (Ns * r), total = rows * nb, B = pass_points(r, P) / r;
    const Div by_nb(nb), by_ns(Ns);
    double2 a[31], o[32];  // (7: two butterflies of a thread)
    for (int u = 0; u < B; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i >= total) continue;
        const int row = rows > 1 ? by_nb(i) : 0, j = i - row * nb;
        const int k = j - by_ns(j) * Ns;
        for (int q = 0; q < r; ++q) {
            a[q] = buf[row * ld + pad8(j + q * nb)];
            if (q > 0 && Ns > 1) a[q] = cmul(a[q], table_at<HALF>(tab, n, q * k * step, sign));
        }
        for (int q = 0; q < r; ++q) {
            double2 sum = a[0];
            int e = 0;  // p q mod r
            for (int p = 1; p < r; ++p) {
                e += q;
                if (e >= r) e -= r;
                sum = cadd(sum, cmul(a[p], table_at<HALF>(tab, n, e * nb, sign)));
            }
            o[u * r + q] = sum;
        }
    }
    __syncthreads();
    for (int u = 0; u < B; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i >= total) continue;
        const int row = rows > 1 ? by_nb(i) : 0, j = i - row * nb;
        const int jq = by_ns(j), k = j - jq * Ns;
        for (int q = 0; q < r; ++q) buf[row * ld + pad8(jq * Ns * r + k + q * Ns)] = o[u * r + q];
    }
    __syncthreads();
}

// the passes over `rows` rows (padded, ld apart) in buf, in place; the CTA has
// at least rows * n / pass_points(r, P) threads for every radix r of the plan
// (fft_threads).  Ends with a block barrier.
template <bool HALF, int P>
__device__ __forceinline__ void smem_fft(double2* buf, const double2* tab, const SmemPlan& S, int sign, int rows, int ld) {
    int Ns = 1;
    for (int s = 0; s < S.nrad; ++s) {
        const int r = S.rad[s];
        switch (r) {
            case 2: smem_pass<2, HALF, P>(buf, tab, S.n, Ns, sign, rows, ld); break;
            case 3: smem_pass<3, HALF, P>(buf, tab, S.n, Ns, sign, rows, ld); break;
            case 4: smem_pass<4, HALF, P>(buf, tab, S.n, Ns, sign, rows, ld); break;
            case 5: smem_pass<5, HALF, P>(buf, tab, S.n, Ns, sign, rows, ld); break;
            case 8: smem_pass<8, HALF, P>(buf, tab, S.n, Ns, sign, rows, ld); break;
            case 16: smem_pass<16, HALF, P>(buf, tab, S.n, Ns, sign, rows, ld); break;
            default: smem_pass_prime<HALF, P>(buf, tab, S.n, Ns, r, sign, rows, ld); break;
        }
        Ns *= r;
    }
}

// complex rows of n <= SMEM_FFT_MAX, one per CTA iteration
__global__ void __launch_bounds__(FFT_THREADS, 1) k_fft_smem(const double2* __restrict__ in, double2* out, int M,
                                                          const __grid_constant__ SmemPlan P, int sign) {
    extern __shared__ double2 sfft[];
    double2* a = sfft;
    double2* tab = a + pad8(P.n);
    make_table<false>(tab, P.n);
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        const double2* x = in + (int64_t)m * P.n;
        for (int i = threadIdx.x; i < P.n; i += blockDim.x) a[pad8(i)] = x[i];
        __syncthreads();
        smem_fft<false, 16>(a, tab, P, sign, 1, 0);
        double2* y = out + (int64_t)m * P.n;
        for (int i = threadIdx.x; i < P.n; i += blockDim.x) y[i] = a[pad8(i)];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Longer rows whose length splits as N = N1 N2 with both factors direct
// shared-memory lengths: the four-step transform (Bailey),
//     X[k1 + N1 k2] = sum_n2 W_N2^(n2 k2) W_N^(n2 k1) sum_n1 x[n1 N2 + n2] W_N1^(n1 k1),
// in two launches with the transposes folded into their loads and stores:
// k_fft4_cols transforms cb columns n2 of x (viewed as N1 x N2) per CTA
// iteration, multiplies by the twiddles W_N^(n2 k1) and writes Y[k1][n2];
// k_fft4_rows transforms kb rows k1 of Y and writes X[k1 + N1 k2].  cb and kb
// are powers of two.  A column's twiddles W_N^(n2 k1) are a product of two
// table entries, k1 = 16 a + b, so that a column needs 16 + N1 / 16 sines and
// cosines instead of N1.
// ---------------------------------------------------------------------------
struct Fft4Plan {
    SmemPlan p1, p2;  // column (N1) and row (N2) transforms
    int64_t n;        // N1 N2
    int cb, kb;       // columns / rows per CTA iteration
};

// shared memory of cb columns of N1: the points, the table and the columns'
// twiddles (fine: 16 each, coarse: N1 / 16 + 1 each)
__host__ __device__ __forceinline__ int cols_tw(int n1) { return 16 + n1 / 16 + 1; }
__host__ __device__ __forceinline__ size_t cols_smem(int n1, int cb) {
    return ((size_t)(cb + 1) * pad8(n1 + 8) + (size_t)cb * cols_tw(n1)) * sizeof(double2);
}

// the twiddles of columns c0 .. c0 + cb - 1: tw[c][b] = W_N^(n2 b), tw[c][16 + a] = W_N^(16 n2 a)
// (exponents below N: no reduction); visible after the caller's barrier
__device__ __forceinline__ void make_col_twiddles(double2* tw, int n1, int cb, int64_t c0, int64_t N) {
    const int per = cols_tw(n1);
    for (int i = threadIdx.x; i < cb * per; i += blockDim.x) {
        const int c = i / per, e = i - c * per;
        const int64_t m = (c0 + c) * (e < 16 ? e : 16 * (e - 16));
        double sv, cv;
        sincospi(2.0 * ((double)m / (double)N), &sv, &cv);
        tw[i] = make_double2(cv, sv);
    }
}
__device__ __forceinline__ double2 col_twiddle(const double2* tw, int n1, int c, int k1, int sign) {
    const double2* t = tw + c * cols_tw(n1);
    const double2 v = cmul(t[k1 & 15], t[16 + (k1 >> 4)]);
    return make_double2(v.x, sign < 0 ? -v.y : v.y);
}

__global__ void __launch_bounds__(FFT_THREADS, 1) k_fft4_cols(const double2* __restrict__ in, double2* Y, int M,
                                                           const __grid_constant__ Fft4Plan F, int sign) {
    extern __shared__ double2 sfft[];
    const int N1 = F.p1.n, N2 = F.p2.n, CB = F.cb, ld = pad8(N1 + 8), lg = __ffs(CB) - 1;
    const int64_t N = F.n;
    double2* a = sfft;
    double2* tab = a + CB * ld;
    double2* tw = tab + ld;
    make_table<false>(tab, N1);
    const int nblk = (N2 + CB - 1) / CB;
    for (int64_t blk = blockIdx.x; blk < (int64_t)M * nblk; blk += gridDim.x) {
        const int64_t m = blk / nblk;
        const int c0 = (int)(blk % nblk) * CB;
        const int cb = min(CB, N2 - c0);
        make_col_twiddles(tw, N1, cb, c0, N);
        for (int i = threadIdx.x; i < N1 << lg; i += blockDim.x) {
            const int n1 = i >> lg, c = i & (CB - 1);
            a[c * ld + pad8(n1)] = c < cb ? in[m * N + (int64_t)n1 * N2 + c0 + c] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        smem_fft<false, 16>(a, tab, F.p1, sign, CB, ld);
        for (int i = threadIdx.x; i < N1 << lg; i += blockDim.x) {
            const int k1 = i >> lg, c = i & (CB - 1);
            if (c < cb) Y[m * N + (int64_t)k1 * N2 + c0 + c] = cmul(a[c * ld + pad8(k1)], col_twiddle(tw, N1, c, k1, sign));
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(FFT_THREADS, 1) k_fft4_rows(const double2* __restrict__ Y, double2* X, int M,
                                                           const __grid_constant__ Fft4Plan F, int sign) {
    extern __shared__ double2 sfft[];
    const int N1 = F.p1.n, N2 = F.p2.n, KB = F.kb, ld = pad8(N2 + 8), lg = __ffs(KB) - 1;
    const int64_t N = F.n;
    double2* a = sfft;
    double2* tab = a + KB * ld;
    make_table<false>(tab, N2);
    const int nblk = (N1 + KB - 1) / KB;
    const Div by_n2(N2);
    for (int64_t blk = blockIdx.x; blk < (int64_t)M * nblk; blk += gridDim.x) {
        const int64_t m = blk / nblk;
        const int k0 = (int)(blk % nblk) * KB;
        const int kb = min(KB, N1 - k0);
        for (int i = threadIdx.x; i < KB * N2; i += blockDim.x) {
            const int kk = by_n2(i), n2 = i - kk * N2;
            a[kk * ld + pad8(n2)] = kk < kb ? Y[m * N + (int64_t)(k0 + kk) * N2 + n2] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        smem_fft<false, 16>(a, tab, F.p2, sign, KB, ld);
        for (int i = threadIdx.x; i < N2 << lg; i += blockDim.x) {
            const int k2 = i >> lg, kk = i & (KB - 1);
            if (kk < kb) X[m * N + k0 + kk + (int64_t)N1 * k2] = a[kk * ld + pad8(k2)];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// The Hilbert transform of real rows, H x = x (*) h circularly over the row,
// through real transforms of an even length L = 2 h: the row is read as h
// complex points z[n] = x[2n] + i x[2n+1], and for each bin pair k, h - k
//     X[k] = E + w O,  X[h-k] = conj(E - w O),   E = (Z[k] + conj Z[h-k]) / 2,
//     O = -i (Z[k] - conj Z[h-k]) / 2,  w = exp(-pi i k / h),
// are multiplied by the transform i g[k] of the (odd, real) kernel and put back
// together the same way.  Half the points of a complex transform of the row,
// and the analytic signal's real part is the row itself.
//   L = N, g = -1 (0 at DC and Nyquist): N even with N / 2 a direct length;
//   L >= 2N - 1 a product of 2, 3 and 5, g from one transform of the kernel:
//     any other N (the circular convolution over N as a linear one: the kernel
//     is known in closed form, so no chirps and two transforms instead of
//     Bluestein's four).
// A long row takes three launches of the four-step transform's two halves:
// columns, rows (transform, multiply and transform back: both bins of a pair
// lie in rows k1 and N1 - k1, which one CTA holds), columns back.  Rows of
// h <= HIL_SMALL points take one launch.
// Against complex transforms of the rows, Bluestein's for a length with a large
// prime factor (B200): 10 rows of 441 003 samples 3790 -> 421 us, 10 of 441 000
// 1367 -> 407 us, 8 of 48 000 78 -> 42 us, 16 of 4963 224 -> 47 us.
// ---------------------------------------------------------------------------
constexpr int HIL_SMALL = 2048;

struct HilPlan {
    SmemPlan p1, p2;  // columns (N1) and rows (N2); one launch: p2 alone
    int64_t h;        // complex points (L / 2)
    int64_t N;        // samples per row
    int cb, ub;       // columns / row pairs per CTA iteration
    int conv;         // 1: L > N, g from the kernel's transform
};

// the circular Hilbert kernel of length N at 0 <= n < N (an odd function of n mod N):
//   N even: (2/N) cot(pi n / N) at odd n, 0 at even n
//   N odd:  (1/N) cot(pi n / 2N) at odd n, -(1/N) tan(pi n / 2N) at even n
// with the argument folded so that its sine or cosine is never formed near a zero
__device__ __forceinline__ double hil_kernel(int64_t n, int64_t N) {
    if (n == 0) return 0.0;
    double sv, cv;
    if ((N & 1) == 0) {
        if ((n & 1) == 0) return 0.0;
        const int64_t m = 2 * n <= N ? n : N - n;  // cot(pi - t) = -cot t
        sincospi((double)m / (double)N, &sv, &cv);
        const double v = (2.0 / (double)N) * (cv / sv);
        return 2 * n <= N ? v : -v;
    }
    // tan t = cot(pi/2 - t): m = n or N - n, the one up to N / 2
    const bool lo = 2 * n <= N;
    sincospi((double)(lo ? n : N - n) / (double)(2 * N), &sv, &cv);
    const double inv = 1.0 / (double)N;
    if (n & 1) return inv * (lo ? cv / sv : sv / cv);
    return -inv * (lo ? sv / cv : cv / sv);
}

// complex point n (samples 2n, 2n+1) of a row's zero-extended samples, or of the kernel
__device__ __forceinline__ double2 hil_point(const double* x, int64_t N, int64_t L, int64_t n) {
    double v[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int64_t t = 2 * n + e;
        if (x) v[e] = t < N ? x[t] : 0.0;
        else v[e] = t < N ? hil_kernel(t, N) : (t > L - N ? -hil_kernel(L - t, N) : 0.0);
    }
    return make_double2(v[0], v[1]);
}

// the pair (k, h - k), k > 0: Z -> W in place (a = Z[k], b = Z[h-k]), with g[k], g[h-k] and w
__device__ __forceinline__ void hil_pair(double2& a, double2& b, double g0, double g1, double2 w) {
    const double2 E = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    const double2 O = make_double2(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));
    const double2 wO = cmul(w, O);
    const double2 Xk = cadd(E, wO), Xm = csub(E, wO);           // X[k], conj X[h-k]
    const double2 c = make_double2(-g0 * Xk.y, g0 * Xk.x);      // Y[k] = i g0 X[k]
    const double2 d = make_double2(g1 * Xm.y, -g1 * Xm.x);      // conj Y[h-k] = -i g1 (E - wO)
    const double2 Ye = make_double2(0.5 * (c.x + d.x), 0.5 * (c.y + d.y));
    const double2 Yo = cmul(make_double2(0.5 * (c.x - d.x), 0.5 * (c.y - d.y)), make_double2(w.x, -w.y));
    a = make_double2(Ye.x - Yo.y, Ye.y + Yo.x);                 // W[k] = Ye + i Yo
    b = make_double2(Ye.x + Yo.y, Yo.x - Ye.y);                 // W[h-k] = conj(Ye) + i conj(Yo)
}

// Im X[k], Im X[h-k] of the same pair
__device__ __forceinline__ double2 hil_imag(double2 a, double2 b, double2 w) {
    const double2 E = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    const double2 wO = cmul(w, make_double2(0.5 * (a.y + b.y), -0.5 * (a.x - b.x)));
    return make_double2(E.y + wO.y, -(E.y - wO.y));
}

// columns: forward from the samples into Y[m][k1][n2] and, where g takes a
// transform, from the kernel into Yk first, or (INV) back from Y into the samples
// of out.  A launch of its own for the kernel was one more latency: 10 rows of
// 441 003 samples 437 -> 421 us, 2 of 100 003 66 -> 57, 9 of 7159 52 -> 46.
template <bool INV, int P>
__global__ void __launch_bounds__(FFT_THREADS, 1) k_hil_cols(const double* x, double2* Y, double2* Yk,
                                                          double* out, int M, const __grid_constant__ HilPlan F) {
    extern __shared__ double2 sfft[];
    const int N1 = F.p1.n, N2 = F.p2.n, CB = F.cb, ld = pad8(N1 + 8), lg = __ffs(CB) - 1;
    double2* a = sfft;
    double2* tab = a + CB * ld;
    double2* tw = tab + ld;
    make_table<false>(tab, N1);
    after_previous_kernel();
    const int nblk = (N2 + CB - 1) / CB, first = !INV && F.conv ? 1 : 0;  // (row 0 is the kernel)
    for (int64_t blk = blockIdx.x; blk < (int64_t)(M + first) * nblk; blk += gridDim.x) {
        const int64_t m = blk / nblk - first;
        const int c0 = (int)(blk % nblk) * CB;
        const int cb = min(CB, N2 - c0);
        const double* xr = INV || m < 0 ? nullptr : x + m * F.N;
        double2* Yr = m < 0 ? Yk : Y + m * F.h;
        make_col_twiddles(tw, N1, cb, c0, F.h);
        if (INV) __syncthreads();
        for (int i = threadIdx.x; i < N1 << lg; i += blockDim.x) {
            const int n1 = i >> lg, c = i & (CB - 1);
            double2 v = make_double2(0.0, 0.0);
            if (c < cb) {
                const int64_t n = (int64_t)n1 * N2 + c0 + c;
                if (INV) v = cmul(Yr[n], col_twiddle(tw, N1, c, n1, +1));  // (n1 is k1 here)
                else v = hil_point(xr, F.N, 2 * F.h, n);
            }
            a[c * ld + pad8(n1)] = v;
        }
        __syncthreads();
        smem_fft<false, P>(a, tab, F.p1, INV ? +1 : -1, CB, ld);
        for (int i = threadIdx.x; i < N1 << lg; i += blockDim.x) {
            const int k1 = i >> lg, c = i & (CB - 1);
            if (c >= cb) continue;
            const int64_t n = (int64_t)k1 * N2 + c0 + c;
            const double2 v = a[c * ld + pad8(k1)];
            if (INV) {
                double* o = out + m * F.N + 2 * n;
                if (2 * n < F.N) o[0] = v.x;
                if (2 * n + 1 < F.N) o[1] = v.y;
            } else {
                Yr[n] = cmul(v, col_twiddle(tw, N1, c, k1, -1));
            }
        }
        __syncthreads();
    }
}

// Row pairs (k1, N1 - k1) of Y: transform, multiply, transform back in place;
// with SPEC the kernel's own row pairs: transform and write g (with the 1 / h
// of the way back).  Unit u = k1 of 0 .. N1 / 2; rows 0 and N1 / 2 pair their
// own bins.
template <bool SPEC, int P>
__global__ void __launch_bounds__(FFT_THREADS, 1) k_hil_rows(double2* Y, double* g, int M,
                                                          const __grid_constant__ HilPlan F) {
    extern __shared__ double2 sfft[];
    const int N1 = F.p1.n, N2 = F.p2.n, UB = F.ub, ld = pad8(N2 + 8), rows = 2 * UB;
    double2* a = sfft;
    double2* half = a + rows * ld;  // exp(pi i m / N2)
    double2* wu = half + ld;        // exp(pi i k1 / h) of each unit
    make_table<true>(half, N2);
    after_previous_kernel();
    const int units = N1 / 2 + 1, nblk = (units + UB - 1) / UB;
    const Div by_n2(N2);
    const double inv = 1.0 / (double)F.h;
    for (int64_t blk = blockIdx.x; blk < (int64_t)M * nblk; blk += gridDim.x) {
        const int64_t m = blk / nblk;
        const int u0 = (int)(blk % nblk) * UB;
        double2* y = Y + m * F.h;
        // buffer row 2q is row u0 + q, row 2q + 1 its mirror (unused where there is none)
        auto row_of = [&](int r) {
            const int u = u0 + (r >> 1);
            if (u >= units) return -1;
            if (!(r & 1)) return u;
            return (u == 0 || 2 * u == N1) ? -1 : N1 - u;
        };
        for (int i = threadIdx.x; i < rows * N2; i += blockDim.x) {
            const int r = by_n2(i), n2 = i - r * N2, k1 = row_of(r);
            a[r * ld + pad8(n2)] = k1 >= 0 ? y[(int64_t)k1 * N2 + n2] : make_double2(0.0, 0.0);
        }
        if (threadIdx.x < UB) {
            double sv, cv;
            sincospi((double)(u0 + (int)threadIdx.x) / (double)F.h, &sv, &cv);
            wu[threadIdx.x] = make_double2(cv, sv);
        }
        __syncthreads();
        smem_fft<true, P>(a, half, F.p2, -1, rows, ld);
        for (int i = threadIdx.x; i < UB * N2; i += blockDim.x) {
            const int q = by_n2(i), k2 = i - q * N2, u = u0 + q;
            if (u >= units) continue;
            const bool own = u == 0 || 2 * u == N1;  // the mirror bin lies in the same row
            const int km = u == 0 ? (k2 ? N2 - k2 : 0) : N2 - 1 - k2;
            if (own && km < k2) continue;
            double2* za = a + (2 * q) * ld + pad8(k2);
            double2* zb = a + (2 * q + (own ? 0 : 1)) * ld + pad8(km);
            const int64_t k = u + (int64_t)N1 * k2;
            const double2 w0 = cmul(wu[q], half[pad8(k2)]);
            const double2 w = make_double2(w0.x, -w0.y);
            if (SPEC) {
                const double2 gi = hil_imag(*za, *zb, w);
                if (k > 0) {
                    g[k] = gi.x * inv;
                    g[F.h - k] = gi.y * inv;
                }
            } else if (k == 0) {
                *za = make_double2(0.0, 0.0);  // DC and Nyquist
            } else {
                double2 va = *za, vb = *zb;
                const double g0 = F.conv ? g[k] : -inv, g1 = F.conv ? g[F.h - k] : -inv;
                hil_pair(va, vb, g0, g1, w);
                *za = va;
                if (!(own && km == k2)) *zb = vb;
            }
        }
        __syncthreads();
        if (!SPEC) {
            smem_fft<true, P>(a, half, F.p2, +1, rows, ld);
            for (int i = threadIdx.x; i < rows * N2; i += blockDim.x) {
                const int rr = by_n2(i), n2 = i - rr * N2, k1 = row_of(rr);
                if (k1 >= 0) y[(int64_t)k1 * N2 + n2] = a[rr * ld + pad8(n2)];
            }
            __syncthreads();
        }
    }
}

// frequency of a sample from the phases (p[-1], p[0], p[1]) as np.gradient of
// the unwrapped phase: one-sided at the row's ends
__device__ __forceinline__ double gradient(double pl, double p, double pr, bool first, bool last, double sr) {
    double f;
    if (first) f = unwrap_diff(pr - p) * sr;
    else if (last) f = unwrap_diff(p - pl) * sr;
    else f = (unwrap_diff(p - pl) + unwrap_diff(pr - p)) * sr * 0.5;
    return f * (0.5 / PI);
}

// arg(z) of a sample.  A zero sample counts as +0 whatever its sign, as a sum
// over a transform's terms gives it: where the row and its transform are zero
// the phase is then zero too (a negative zero would make it +-pi).
__device__ __forceinline__ double phase_of(double re, double im) { return atan2(im, re + 0.0); }

// |z| of a sample: the root of the squares' sum where they neither overflow nor
// underflow, hypot elsewhere; a row with a non-finite sample has no finite
// transform, so its magnitude is not a number throughout, as with a transform
// of the row
__device__ __forceinline__ double magnitude(double re, double im) {
    const double q = fma(re, re, im * im);
    if (q > 1e-280 && q < 1e280) return sqrt(q);
    return isnan(im) ? im : hypot(re, im);
}

// frequency and amplitude from the rows and their Hilbert transforms: every
// phase is formed once (and twice at a tile's two ends), not by each of the
// three samples that read it; bound by the arc tangents' instructions
constexpr int IF_THREADS = 256, IF_TILE = 4 * IF_THREADS;
__global__ void __launch_bounds__(IF_THREADS) k_hil_out(const double* x, const double* hx,
                                                        double* inst_freq, double* inst_amp, int M, int64_t N,
                                                        double sr) {
    __shared__ double ph[IF_TILE + 2];
    after_previous_kernel();
    const int64_t tiles = (N + IF_TILE - 1) / IF_TILE;
    for (int64_t blk = blockIdx.x; blk < (int64_t)M * tiles; blk += gridDim.x) {
        const int64_t m = blk / tiles, t0 = (blk % tiles) * IF_TILE;
        const int n = (int)min((int64_t)IF_TILE, N - t0);
        const double* xr = x + m * N + t0;
        const double* hr = hx + m * N + t0;
        for (int i = threadIdx.x; i < n; i += IF_THREADS) ph[i + 1] = phase_of(xr[i], hr[i]);
        if (threadIdx.x == IF_THREADS - 1 && t0 > 0) ph[0] = phase_of(xr[-1], hr[-1]);
        if (threadIdx.x == IF_THREADS - 33 && t0 + n < N) ph[n + 1] = phase_of(xr[n], hr[n]);
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += IF_THREADS) {
            const int64_t t = t0 + i;
            inst_freq[m * N + t] = gradient(ph[i], ph[i + 1], ph[i + 2], t == 0, t == N - 1, sr);
            inst_amp[m * N + t] = magnitude(xr[i], hr[i]);
        }
        __syncthreads();
    }
}

// h <= HIL_SMALL: the whole row in one CTA iteration (g: the kernel's transform
// from a launch with x null and M = 1, or unread when L = N)
template <bool SPEC, int P>
__global__ void __launch_bounds__(FFT_THREADS, 1) k_hil_small(const double* x, double* g, double* inst_freq,
                                                           double* inst_amp, int M, double sr,
                                                           const __grid_constant__ HilPlan F) {
    extern __shared__ double2 sfft[];
    const int h = F.p2.n, ld = pad8(h + 8), N = (int)F.N;
    double2* a = sfft;
    double2* half = a + ld;
    double* ph = reinterpret_cast<double*>(half + ld);  // phases (N <= 2h)
    make_table<true>(half, h);
    after_previous_kernel();
    const double inv = 1.0 / (double)h;
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        const double* xr = SPEC ? nullptr : x + (int64_t)m * N;
        for (int i = threadIdx.x; i < h; i += blockDim.x) a[pad8(i)] = hil_point(xr, N, 2 * (int64_t)h, i);
        __syncthreads();
        smem_fft<true, P>(a, half, F.p2, -1, 1, 0);
        for (int k = threadIdx.x; 2 * k <= h; k += blockDim.x) {
            double2* za = a + pad8(k);
            double2* zb = a + pad8(k ? h - k : 0);
            const double2 w0 = half[pad8(k)], w = make_double2(w0.x, -w0.y);
            if (SPEC) {
                const double2 gi = hil_imag(*za, *zb, w);
                if (k > 0) {
                    g[k] = gi.x * inv;
                    g[h - k] = gi.y * inv;
                }
            } else if (k == 0) {
                // (zero, and not a number where a sample is not finite: the only bin of two samples)
                const double z = (za->x - za->x) + (za->y - za->y);
                *za = make_double2(z, z);
            } else {
                double2 va = *za, vb = *zb;
                hil_pair(va, vb, F.conv ? g[k] : -inv, F.conv ? g[h - k] : -inv, w);
                *za = va;
                if (2 * k != h) *zb = vb;
            }
        }
        __syncthreads();
        if (!SPEC) {
            smem_fft<true, P>(a, half, F.p2, +1, 1, 0);
            auto im_at = [&](int t) { return (t & 1) ? a[pad8(t >> 1)].y : a[pad8(t >> 1)].x; };
            for (int t = threadIdx.x; t < N; t += blockDim.x) ph[t] = phase_of(xr[t], im_at(t));
            __syncthreads();
            for (int t = threadIdx.x; t < N; t += blockDim.x) {
                inst_freq[(int64_t)m * N + t] = gradient(t > 0 ? ph[t - 1] : 0.0, ph[t], t + 1 < N ? ph[t + 1] : 0.0,
                                                         t == 0, t == N - 1, sr);
                inst_amp[(int64_t)m * N + t] = magnitude(xr[t], im_at(t));
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// STFT of frames whose length is a direct shared-memory length.  EVEN: the
// windowed frame is read as h = nperseg / 2 complex points and its one-sided
// bins follow from their transform (as above: X[k] = E + w O), half the work
// and space of a complex transform; odd lengths (h = nperseg) transform the
// frame as it is.  A CTA takes fb consecutive frames of a row at a time, so that
// bin f of frames j .. j + fb - 1 is one contiguous store of Z[m][f][.] (16 bytes
// per frame).  The window 0.5 - 0.5 cos(2 pi n / nperseg) and w come from the
// transform's own half-step table.  Bound by shared-memory wavefronts (55 % of
// their rate) and latency.  11 rows of 480 000 samples in frames of 4096: 366 us
// with one frame per 1024-thread CTA in 192 KB (complex, six passes), 100 us
// with two frames per 256-thread CTA in 111 KB; 12 rows of a million samples in
// frames of 512: 2126 -> 138 us.
// ---------------------------------------------------------------------------
struct StftPlan {
    SmemPlan p;  // h points
    int step, T, fb;
};

template <bool EVEN, int P>
__global__ void __launch_bounds__(FFT_THREADS, 1) k_stft(const double* __restrict__ x, double2* Z, int M, int64_t N,
                                                      double inv_wsum, const __grid_constant__ StftPlan S) {
    extern __shared__ double2 sfft[];
    const int h = S.p.n, ld = pad8(h + 8), FB = S.fb, lg = __ffs(FB) - 1, T = S.T;
    const int nperseg = EVEN ? 2 * h : h, F = nperseg / 2 + 1;
    double2* a = sfft;
    double2* half = a + FB * ld;  // exp(pi i m / h), m < h
    make_table<true>(half, h);
    __syncthreads();
    const int nblk = (T + FB - 1) / FB;
    const Div by_h(h);
    // sample s of a row under window position q: cos(2 pi q / nperseg) is entry q
    // (even lengths) or 2 q of the table, the second half turn by its sign
    auto windowed = [&](const double* xr, int64_t s, int q) {
        const int e = EVEN ? q : 2 * q;
        const double c = e < h ? half[pad8(e)].x : -half[pad8(e - h)].x;
        return (s >= 0 && s < N) ? xr[s] * (0.5 - 0.5 * c) : 0.0;
    };
    for (int64_t blk = blockIdx.x; blk < (int64_t)M * nblk; blk += gridDim.x) {
        const int64_t m = blk / nblk;
        const int j0 = (int)(blk % nblk) * FB;
        const double* xr = x + m * N;
        for (int i = threadIdx.x; i < FB * h; i += blockDim.x) {
            const int f = by_h(i), n = i - f * h;
            const int64_t s0 = (int64_t)(j0 + f) * S.step - nperseg / 2;  // the frame's first sample
            double2 v = make_double2(0.0, 0.0);
            if (j0 + f < T) {
                if (EVEN) v = make_double2(windowed(xr, s0 + 2 * n, 2 * n), windowed(xr, s0 + 2 * n + 1, 2 * n + 1));
                else v.x = windowed(xr, s0 + n, n);
            }
            a[f * ld + pad8(n)] = v;
        }
        __syncthreads();
        smem_fft<true, P>(a, half, S.p, -1, FB, ld);
        if (EVEN) {
            // bins k and h - k of every frame (k = 0: DC and Nyquist)
            for (int i = threadIdx.x; i < (h / 2 + 1) << lg; i += blockDim.x) {
                const int k = i >> lg, f = i & (FB - 1), km = h - k;
                if (j0 + f >= T) continue;
                const double2 za = a[f * ld + pad8(k)], zb = a[f * ld + pad8(k ? km : 0)];
                const double2 E = make_double2(0.5 * (za.x + zb.x), 0.5 * (za.y - zb.y));
                const double2 O = make_double2(0.5 * (za.y + zb.y), -0.5 * (za.x - zb.x));
                const double2 w = half[pad8(k)];
                const double2 wO = cmul(make_double2(w.x, -w.y), O);
                double2* z = Z + (m * F + k) * T + j0 + f;
                double2* zm = Z + (m * F + km) * T + j0 + f;
                *z = make_double2((E.x + wO.x) * inv_wsum, (E.y + wO.y) * inv_wsum);
                if (km != k) *zm = make_double2((E.x - wO.x) * inv_wsum, -(E.y - wO.y) * inv_wsum);
            }
        } else {
            for (int i = threadIdx.x; i < F << lg; i += blockDim.x) {
                const int k = i >> lg, f = i & (FB - 1);
                if (j0 + f >= T) continue;
                const double2 v = a[f * ld + pad8(k)];
                Z[(m * F + k) * T + j0 + f] = make_double2(v.x * inv_wsum, v.y * inv_wsum);
            }
        }
        __syncthreads();
    }
}


// Bluestein: chirp c_n = exp(sign pi i n^2 / N) (n^2 reduced mod 2N exactly)
__device__ __forceinline__ double2 chirp(int64_t n, int64_t N, int sign) {
    const int64_t r = (int64_t)(((unsigned long long)n * (unsigned long long)n) % (unsigned long long)(2 * N));
    double s, c;
    sincospi((double)r / (double)N, &s, &c);
    return make_double2(c, sign < 0 ? -s : s);
}

// a[m][n] = x[m][n] c_n for n < N, 0 up to L
__global__ void k_blue_pre(const double2* __restrict__ x, double2* a, int M, int64_t N, int64_t L, int sign) {
    const int64_t total = (int64_t)M * L;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = i / L, n = i % L;
        a[i] = n < N ? cmul(x[m * N + n], chirp(n, N, sign)) : make_double2(0.0, 0.0);
    }
}

// b[n] = conj(c_n) for n < N, b[L-n] = conj(c_n) for 0 < n < N, 0 elsewhere
__global__ void k_blue_kernel(double2* b, int64_t N, int64_t L, int sign) {
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < L; n += (int64_t)gridDim.x * blockDim.x) {
        double2 v = make_double2(0.0, 0.0);
        if (n < N) v = chirp(n, N, -sign);
        else if (L - n < N) v = chirp(L - n, N, -sign);
        b[n] = v;
    }
}

// A[m][n] *= B[n] / L
__global__ void k_blue_mul(double2* A, const double2* __restrict__ B, int M, int64_t L) {
    const int64_t total = (int64_t)M * L;
    const double inv = 1.0 / (double)L;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double2 v = cmul(A[i], B[i % L]);
        A[i] = make_double2(v.x * inv, v.y * inv);
    }
}

// y[m][k] = c_k C[m][k] for k < N
__global__ void k_blue_post(const double2* __restrict__ Cv, double2* y, int M, int64_t N, int64_t L, int sign) {
    const int64_t total = (int64_t)M * N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = i / N, k = i % N;
        y[i] = cmul(Cv[m * L + k], chirp(k, N, sign));
    }
}

struct FftPlan {
    int64_t n = 0, L = 0;        // length; Bluestein's power-of-two length (0 = direct)
    std::vector<int> radices;    // of n (direct) or of L (Bluestein)
};

bool factor(int64_t n, std::vector<int>& rad) {
    rad.clear();
    while (n % 4 == 0) { rad.push_back(4); n /= 4; }
    while (n % 2 == 0) { rad.push_back(2); n /= 2; }
    for (int p = 3; p <= 31; p += 2) {
        while (n % p == 0) { rad.push_back(p); n /= p; }
    }
    return n == 1;
}

FftPlan make_fft_plan(int64_t n) {
    FftPlan P;
    P.n = n;
    if (!factor(n, P.radices)) {
        int64_t L = 1;
        while (L < 2 * n - 1) L <<= 1;
        P.L = L;
        factor(L, P.radices);
    }
    return P;
}

// complex elements of scratch an FFT of M rows needs beyond its two ping-pong buffers
int64_t fft_extra(const FftPlan& P, int M) { return P.L ? 2 * (int64_t)M * P.L + 2 * P.L : 0; }

// largest dynamic shared memory of a CTA
constexpr int SMEM_LIMIT = 227 * 1024;

// the shared-memory plan of a direct length up to SMEM_FFT_MAX: radices 16, 8,
// 4, 2, then 5, 3 and the odd primes up to 31; false when it has a larger factor
bool smem_plan(int64_t len, SmemPlan& sp) {
    if (len < 1 || len > SMEM_FFT_MAX) return false;
    sp.n = (int)len;
    sp.nrad = 0;
    int n = (int)len;
    auto take = [&](int r) {
        sp.rad[sp.nrad++] = r;
        n /= r;
    };
    int two = 0;
    for (int v = n; v % 2 == 0; v /= 2) ++two;
    // 2^two in as few passes as radix 16 allows, the widths evened out (2^9 as 8 8 8, not 16 16 2)
    for (int passes = (two + 3) / 4; passes > 0; --passes) {
        const int w = (two + passes - 1) / passes;
        take(1 << w);
        two -= w;
    }
    while (n % 5 == 0) take(5);
    for (int p = 3; p <= 31; p += 2)
        while (n % p == 0 && sp.nrad < SMEM_FFT_MAXRAD) take(p);
    return n == 1;
}

// a kernel's shared memory limit raised to SMEM_LIMIT (set at each call: an
// attribute of the current device)
bool smem_ready(const void* fn) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) == cudaSuccess;
}

unsigned smem_grid(int64_t rows) { return (unsigned)(rows < 65535 ? rows : 65535); }

// the Hann window's sum, added in index order (as the reference's window sum
// is formed); the last length's sum is kept per thread, since the host loop
// of nperseg cosines costs more than the STFT's launch
double window_sum(int nperseg) {
    thread_local int last_n = 0;
    thread_local double last_sum = 0.0;
    if (nperseg != last_n) {
        double wsum = 0.0;
        for (int n = 0; n < nperseg; ++n) wsum += 0.5 - 0.5 * cos(2.0 * PI * (double)n / (double)nperseg);
        last_n = nperseg;
        last_sum = wsum;
    }
    return last_sum;
}

// CTAs of one wave and its latency: about two per SM
constexpr int64_t FEW_CTAS = 2 * 148;

// threads of a CTA that transforms `rows` rows of a plan at a time
int fft_threads(const SmemPlan& p, int rows, int P) {
    int points = P;
    for (int i = 0; i < p.nrad; ++i) points = std::min(points, pass_points(p.rad[i], P));
    const int t = (rows * p.n + points - 1) / points;
    return std::max(32, (t + 31) / 32 * 32);
}

// CTAs of a kernel of one table per CTA: no more than the SMs hold at a time
// (512 threads of 128 registers each); the CTAs then take their blocks in turn
unsigned persistent_grid(int64_t blocks, int threads, size_t smem) {
    const int64_t per_sm = std::max<int64_t>(1, std::min<int64_t>(FFT_THREADS / threads, SMEM_LIMIT / (int64_t)(smem + 1024)));
    return (unsigned)std::min<int64_t>(blocks, 148 * per_sm);
}

// columns or rows (at most 8, a power of two) of a plan for one CTA iteration:
// as many as keep a CTA at GROUP_POINTS points, so that three CTAs of 128 to
// 256 threads share an SM
constexpr int GROUP_POINTS = 2048;
int group_of(const SmemPlan& p, int others) {
    int g = 8;
    while (g > 1 && (g > others || g * p.n > GROUP_POINTS || fft_threads(p, g, 16) > FFT_THREADS)) g >>= 1;
    return g;
}

// the four-step split of a length: N1 the divisor nearest below sqrt(n) with
// both N1 and n / N1 direct lengths of at most `most`; false when there is none
bool split_plan(int64_t n, int most, SmemPlan& p1, SmemPlan& p2) {
    if (n > (int64_t)most * most) return false;
    int64_t n1 = 1;
    while ((n1 + 1) * (n1 + 1) <= n) ++n1;
    for (; n1 >= 2; --n1) {
        if (n % n1) continue;
        if (n / n1 > most) break;  // n / n1 only grows as n1 shrinks
        if (smem_plan(n1, p1) && smem_plan(n / n1, p2)) return true;
    }
    return false;
}

bool fft4_plan(int64_t n, Fft4Plan& F) {
    if (n <= SMEM_FFT_MAX || !split_plan(n, SMEM_FFT_MAX, F.p1, F.p2)) return false;
    F.n = n;
    F.cb = group_of(F.p1, F.p2.n);
    F.kb = group_of(F.p2, F.p1.n);
    return true;
}

// the two launches of a four-step transform of M rows: in -> y (columns), y -> out (rows)
void fft4(const double2* in, double2* y, double2* out, int M, const Fft4Plan& F, int sign, cudaStream_t st) {
    const int64_t nc = (int64_t)M * ((F.p2.n + F.cb - 1) / F.cb), nr = (int64_t)M * ((F.p1.n + F.kb - 1) / F.kb);
    k_fft4_cols<<<smem_grid(nc), fft_threads(F.p1, F.cb, 16), cols_smem(F.p1.n, F.cb), st>>>(in, y, M, F, sign);
    k_fft4_rows<<<smem_grid(nr), fft_threads(F.p2, F.kb, 16), (size_t)(F.kb + 1) * pad8(F.p2.n + 8) * sizeof(double2), st>>>(
        y, out, M, F, sign);
}

// The plan of the Hilbert transform of rows of N samples, false where it runs
// through complex transforms of the rows (longer than about 8 million samples).
constexpr int HIL_MAXROW = 2048;  // two columns, or a row pair, in 4096 points
bool hil_plan(int64_t N, HilPlan& F) {
    F.N = N;
    F.conv = 0;
    F.cb = F.ub = 1;
    F.p1.n = 1;
    auto long_plan = [&](int64_t h) {
        if (!split_plan(h, HIL_MAXROW, F.p1, F.p2)) return false;
        if (fft_threads(F.p1, 2, 16) > FFT_THREADS || fft_threads(F.p2, 2, 16) > FFT_THREADS) return false;
        F.h = h;
        F.cb = std::max(2, group_of(F.p1, F.p2.n));
        F.ub = std::max(1, group_of(F.p2, F.p1.n) / 2);
        return true;
    };
    // L = N: radix 7 and above are slow enough that a longer 2-3-5 convolution is not worse
    if (N % 2 == 0) {
        const int64_t h = N / 2;
        if (h <= HIL_SMALL && smem_plan(h, F.p2)) {
            F.h = h;
            return true;
        }
        if (h > HIL_SMALL && long_plan(h)) return true;
    }
    // L = 2h >= 2N - 1: the least h = N1 N2 >= N of products of 2, 3 and 5
    F.conv = 1;
    int64_t best = 0;
    if (N <= HIL_SMALL) {
        int64_t h = N;
        auto smooth = [](int64_t v) {
            for (int p : {2, 3, 5})
                while (v % p == 0) v /= p;
            return v == 1;
        };
        while (!smooth(h)) ++h;
        if (h <= HIL_SMALL && smem_plan(h, F.p2)) {
            F.h = h;
            return true;
        }
    }
    // products of 2, 3 and 5 up to HIL_MAXROW, in order
    static const std::vector<int> nice = [] {
        std::vector<int> v;
        for (int a = 1; a <= HIL_MAXROW; a *= 2)
            for (int b = a; b <= HIL_MAXROW; b *= 3)
                for (int c = b; c <= HIL_MAXROW; c *= 5) v.push_back(c);
        std::sort(v.begin(), v.end());
        return v;
    }();
    for (int a : nice) {  // a = N1 <= N2 <= 2 N1 (rows near the columns' length keep more CTAs on an SM)
        const int64_t need = std::max<int64_t>((N + a - 1) / a, a);
        const auto it = std::lower_bound(nice.begin(), nice.end(), need);
        if (it == nice.end() || *it > 2 * a) continue;
        const int64_t h = (int64_t)a * *it;
        if (best == 0 || h < best) {
            best = h;
            smem_plan(a, F.p1);
            smem_plan(*it, F.p2);
        }
    }
    if (best == 0) return false;
    F.h = best;
    F.cb = std::max(2, group_of(F.p1, F.p2.n));
    F.ub = std::max(1, group_of(F.p2, F.p1.n) / 2);
    return true;
}

bool hil_small(const HilPlan& F) { return F.p1.n == 1; }

// whether [a, a + na) and [b, b + nb) share a byte
bool overlaps(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t pa = reinterpret_cast<uintptr_t>(a), pb = reinterpret_cast<uintptr_t>(b);
    return pa < pb + nb && pb < pa + na;
}

// workspace of the plan: Y, the kernel's Y and g, the rows' Hilbert transforms
size_t hil_bytes(const HilPlan& F, int64_t M) {
    const size_t gb = F.conv ? al((size_t)(F.h + 1) * sizeof(double)) : 0;
    if (hil_small(F)) return gb;
    return al((size_t)M * F.h * sizeof(double2)) + al((size_t)M * F.N * sizeof(double)) + gb +
           (F.conv ? al((size_t)F.h * sizeof(double2)) : 0);
}

// a launch that may begin while the stream's previous kernel drains
template <typename... Params, typename... Args>
void launch_after(void (*fn)(Params...), unsigned grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, fn, static_cast<Params>(args)...);  // (the caller reads the last error)
}

template <int P>
int hil_launch(const double* x, int M, double sr, double* freq, double* amp, void* ws, const HilPlan& F,
               cudaStream_t st) {
    char* base = static_cast<char*>(ws);
    double* g = reinterpret_cast<double*>(base);
    if (F.conv) base += al((size_t)(F.h + 1) * sizeof(double));
    if (hil_small(F)) {
        if (!smem_ready(reinterpret_cast<const void*>(k_hil_small<true, P>)) ||
            !smem_ready(reinterpret_cast<const void*>(k_hil_small<false, P>)))
            return EEMD_SP_E_CUDA;
        const size_t sm = (size_t)3 * pad8(F.p2.n + 8) * sizeof(double2);
        const int nt = fft_threads(F.p2, 1, P);
        if (F.conv) launch_after(k_hil_small<true, P>, 1, nt, sm, st, static_cast<double*>(nullptr), g, static_cast<double*>(nullptr), static_cast<double*>(nullptr), 1, sr, F);
        launch_after(k_hil_small<false, P>, smem_grid(M), nt, sm, st, x, g, freq, amp, M, sr, F);
        return EEMD_SP_OK;
    }
    if (!smem_ready(reinterpret_cast<const void*>(k_hil_cols<false, P>)) ||
        !smem_ready(reinterpret_cast<const void*>(k_hil_cols<true, P>)) ||
        !smem_ready(reinterpret_cast<const void*>(k_hil_rows<false, P>)) ||
        !smem_ready(reinterpret_cast<const void*>(k_hil_rows<true, P>)))
        return EEMD_SP_E_CUDA;
    double2* Y = reinterpret_cast<double2*>(base);
    base += al((size_t)M * F.h * sizeof(double2));
    double* hx = reinterpret_cast<double*>(base);
    base += al((size_t)M * F.N * sizeof(double));
    const size_t sc = cols_smem(F.p1.n, F.cb);
    const size_t sr_ = (size_t)(2 * F.ub + 1) * pad8(F.p2.n + 8) * sizeof(double2) + F.ub * sizeof(double2);
    const int tc = fft_threads(F.p1, F.cb, P), tr = fft_threads(F.p2, 2 * F.ub, P);
    const int64_t bc = (F.p2.n + F.cb - 1) / F.cb, br = (F.p1.n / 2 + 1 + F.ub - 1) / F.ub;
    double2* Yk = reinterpret_cast<double2*>(base);  // (conv)
    launch_after(k_hil_cols<false, P>, smem_grid(bc * (M + (F.conv ? 1 : 0))), tc, sc, st, x, Y, Yk, static_cast<double*>(nullptr), M, F);
    if (F.conv) launch_after(k_hil_rows<true, P>, smem_grid(br), tr, sr_, st, Yk, g, 1, F);
    launch_after(k_hil_rows<false, P>, smem_grid(br * M), tr, sr_, st, Y, g, M, F);
    launch_after(k_hil_cols<true, P>, smem_grid(bc * M), tc, sc, st, static_cast<double*>(nullptr), Y, static_cast<double2*>(nullptr), hx, M, F);
    launch_after(k_hil_out, smem_grid(((F.N + IF_TILE - 1) / IF_TILE) * M), IF_THREADS, 0, st, x, hx, freq, amp, M, F.N, sr);
    return EEMD_SP_OK;
}

// 8 points per thread where the transforms make no more than about two CTAs per
// SM (and the threads fit a CTA), with smaller groups for more CTAs
int hil_run(const double* x, int M, double sr, double* freq, double* amp, void* ws, HilPlan& F, cudaStream_t st) {
    if (hil_small(F)) {
        if (M <= FEW_CTAS && fft_threads(F.p2, 1, 8) <= FFT_THREADS) return hil_launch<8>(x, M, sr, freq, amp, ws, F, st);
        return hil_launch<16>(x, M, sr, freq, amp, ws, F, st);
    }
    while (F.cb > 2 && (int64_t)M * ((F.p2.n + F.cb - 1) / F.cb) < FEW_CTAS) F.cb >>= 1;
    while (F.ub > 1 && (int64_t)M * ((F.p1.n / 2 + F.ub) / F.ub) < FEW_CTAS) F.ub >>= 1;
    const bool few = (int64_t)M * F.h <= FEW_CTAS * GROUP_POINTS / 2 && fft_threads(F.p1, F.cb, 8) <= FFT_THREADS &&
                     fft_threads(F.p2, 2 * F.ub, 8) <= FFT_THREADS;
    return few ? hil_launch<8>(x, M, sr, freq, amp, ws, F, st) : hil_launch<16>(x, M, sr, freq, amp, ws, F, st);
}

// the fused kernel's plan: frames of a direct length up to SMEM_FFT_MAX
bool stft_plan(int nperseg, int M, int step, int T, StftPlan& S) {
    if (nperseg > SMEM_FFT_MAX || !smem_plan(nperseg % 2 ? nperseg : nperseg / 2, S.p)) return false;
    S.step = step;
    S.T = T;
    // up to 4096 points: two frames of 4096 samples, two CTAs of 111 KB per SM
    S.fb = 8;
    while (S.fb > 1 && (S.fb > T || S.fb * S.p.n > SMEM_FFT_MAX || fft_threads(S.p, S.fb, 16) > FFT_THREADS)) S.fb >>= 1;
    while (S.fb > 1 && (int64_t)M * ((T + S.fb - 1) / S.fb) < FEW_CTAS) S.fb >>= 1;
    return true;
}

// Stockham passes of length len over M rows: src -> (b1, b2 alternately); returns the result buffer
double2* stockham(const double2* src, double2* b1, double2* b2, int M, int64_t len, const std::vector<int>& rad,
                  int sign, cudaStream_t st) {
    const double2* cur = src;
    double2* dst = b1;
    int64_t Ns = 1;
    if (rad.empty()) {  // length 1: the transform is the identity
        cudaMemcpyAsync(b1, src, sizeof(double2) * (size_t)M * (size_t)len, cudaMemcpyDeviceToDevice, st);
        return b1;
    }
    SmemPlan sp;
    if (len <= SMEM_FFT_MAX && smem_plan(len, sp) && smem_ready(reinterpret_cast<const void*>(k_fft_smem))) {
        k_fft_smem<<<smem_grid(M), fft_threads(sp, 1, 16), 2 * pad8(sp.n) * sizeof(double2), st>>>(src, b1, M, sp, sign);
        return b1;
    }
    Fft4Plan f4;
    if (fft4_plan(len, f4) && smem_ready(reinterpret_cast<const void*>(k_fft4_cols)) &&
        smem_ready(reinterpret_cast<const void*>(k_fft4_rows))) {
        // src -> b1 (columns), b1 -> b2 (rows): b2 may be src, which only the first launch reads
        fft4(src, b1, b2, M, f4, sign, st);
        return b2;
    }
    for (int r : rad) {
        const unsigned g = grid_for((int64_t)M * (len / r));
        switch (r) {
            case 2: k_fft_pass<2><<<g, 256, 0, st>>>(cur, dst, M, len, Ns, sign); break;
            case 3: k_fft_pass<3><<<g, 256, 0, st>>>(cur, dst, M, len, Ns, sign); break;
            case 4: k_fft_pass<4><<<g, 256, 0, st>>>(cur, dst, M, len, Ns, sign); break;
            case 5: k_fft_pass<5><<<g, 256, 0, st>>>(cur, dst, M, len, Ns, sign); break;
            default: k_fft_pass_prime<<<g, 256, 0, st>>>(cur, dst, M, len, Ns, r, sign); break;
        }
        Ns *= r;
        cur = dst;
        dst = (dst == b1) ? b2 : b1;
    }
    return const_cast<double2*>(cur);
}

// FFT of M rows of length P.n: `in` is read only; b1, b2 hold M*n each and
// `extra` fft_extra(P, M) elements; returns the buffer (b1 or b2) with the result
double2* fft_rows(const double2* in, double2* b1, double2* b2, double2* extra, int M, const FftPlan& P, int sign,
                  cudaStream_t st) {
    if (!P.L) return stockham(in, b1, b2, M, P.n, P.radices, sign, st);
    const int64_t N = P.n, L = P.L;
    double2* A = extra;                 // M * L
    double2* T = extra + (int64_t)M * L;  // M * L
    double2* Bk = T + (int64_t)M * L;   // L
    double2* Bt = Bk + L;               // L
    k_blue_pre<<<grid_for((int64_t)M * L), 256, 0, st>>>(in, A, M, N, L, sign);
    k_blue_kernel<<<grid_for(L), 256, 0, st>>>(Bk, N, L, sign);
    double2* Af = stockham(A, T, A, M, L, P.radices, -1, st);
    double2* Bf = stockham(Bk, Bt, Bk, 1, L, P.radices, -1, st);
    k_blue_mul<<<grid_for((int64_t)M * L), 256, 0, st>>>(Af, Bf, M, L);
    double2* other = (Af == A) ? T : A;
    double2* Cv = stockham(Af, other, Af, M, L, P.radices, +1, st);
    k_blue_post<<<grid_for((int64_t)M * N), 256, 0, st>>>(Cv, b1, M, N, L, sign);
    return b1;
}

// three complex buffers of `rows` x `len` plus the FFT's extra scratch
struct FftLayout {
    FftPlan P;
    int64_t rows = 0;
    size_t buf = 0, extra = 0, total = 0;
};

int fft_layout(int64_t rows, int64_t len, FftLayout& L) {
    if (rows < 1 || len < 1 || rows > (1LL << 31)) return EEMD_SP_E_BADARG;
    L.P = make_fft_plan(len);
    L.rows = rows;
    L.buf = al((size_t)rows * (size_t)len * sizeof(double2));
    L.extra = al((size_t)fft_extra(L.P, (int)rows) * sizeof(double2));
    L.total = 3 * L.buf + L.extra;
    return EEMD_SP_OK;
}

struct Bufs {
    double2 *x, *y, *z, *extra;
};

Bufs carve(void* ws, const FftLayout& L) {
    char* base = static_cast<char*>(ws);
    Bufs b;
    b.x = reinterpret_cast<double2*>(base);
    b.y = reinterpret_cast<double2*>(base + L.buf);
    b.z = reinterpret_cast<double2*>(base + 2 * L.buf);
    b.extra = reinterpret_cast<double2*>(base + 3 * L.buf);
    return b;
}

int stft_shape(int64_t N, int nperseg, int noverlap, int& F, int& T) {
    if (N < 1 || nperseg < 2 || noverlap < 0 || noverlap >= nperseg) return EEMD_SP_E_BADARG;
    const int64_t ext = N + 2 * (int64_t)(nperseg / 2);
    if (ext < nperseg) return EEMD_SP_E_BADARG;
    const int64_t t = (ext - noverlap) / (nperseg - noverlap);
    if (t < 1 || t > (1LL << 30)) return EEMD_SP_E_BADARG;
    F = nperseg / 2 + 1;
    T = (int)t;
    return EEMD_SP_OK;
}

}  // namespace sp

using namespace sp;

extern "C" {

int32_t eemd_sp_version(void) { return EEMD_SP_ABI_VERSION; }

int32_t eemd_sp_fft_workspace(int32_t M, int64_t N, size_t* bytes) {
    if (!bytes) return EEMD_SP_E_BADARG;
    FftLayout L;
    const int rc = fft_layout(M, N, L);
    if (rc) return rc;
    *bytes = L.total;
    return EEMD_SP_OK;
}

int32_t eemd_sp_fft(const double* in, double* out, int32_t M, int64_t N, int32_t sign, void* ws, size_t ws_bytes,
                    void* stream) {
    if (!in || !out || !ws || (sign != -1 && sign != 1)) return EEMD_SP_E_BADARG;
    FftLayout L;
    int rc = fft_layout(M, N, L);
    if (rc) return rc;
    if (ws_bytes < L.total) return EEMD_SP_E_NOMEM;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Bufs b = carve(ws, L);
    const size_t nb = sizeof(double2) * (size_t)M * (size_t)N;
    if (cudaMemcpyAsync(b.x, in, nb, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return EEMD_SP_E_CUDA;
    double2* r = fft_rows(b.x, b.y, b.z, b.extra, M, L.P, sign, st);
    if (cudaMemcpyAsync(out, r, nb, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return EEMD_SP_E_CUDA;
    return cudaGetLastError() == cudaSuccess ? EEMD_SP_OK : EEMD_SP_E_CUDA;
}

int32_t eemd_sp_hilbert_workspace(int32_t M, int64_t N, size_t* bytes) {
    if (!bytes || N < 2) return EEMD_SP_E_BADARG;
    const int rc = eemd_sp_fft_workspace(M, N, bytes);  // of the complex transforms; checks M and N
    if (rc) return rc;
    HilPlan F;
    if (hil_plan(N, F)) *bytes = std::max(*bytes, hil_bytes(F, M));
    return EEMD_SP_OK;
}

int32_t eemd_sp_hilbert_if(const double* x, int32_t M, int64_t N, double sr, double* inst_freq, double* inst_amp,
                           void* ws, size_t ws_bytes, void* stream) {
    if (!x || !inst_freq || !inst_amp || !ws || !(sr > 0.0) || N < 2) return EEMD_SP_E_BADARG;
    FftLayout L;
    int rc = fft_layout(M, N, L);
    if (rc) return rc;
    if (ws_bytes < L.total) return EEMD_SP_E_NOMEM;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Bufs b = carve(ws, L);
    const int64_t total = (int64_t)M * N;
    // the real transforms' last kernel reads the rows (and a tile's neighbours) while it
    // writes the outputs: rows that share memory with an output are copied first
    const size_t nb = sizeof(double) * (size_t)total;
    const bool in_place = overlaps(x, nb, inst_freq, nb) || overlaps(x, nb, inst_amp, nb);
    const size_t copy = in_place ? al(nb) : 0;
    HilPlan F;
    if (hil_plan(N, F) && copy + hil_bytes(F, M) <= ws_bytes) {
        if (in_place) {
            if (cudaMemcpyAsync(ws, x, nb, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return EEMD_SP_E_CUDA;
            x = static_cast<const double*>(ws);
            ws = static_cast<char*>(ws) + copy;
        }
        const int r = hil_run(x, M, sr, inst_freq, inst_amp, ws, F, st);
        if (r) return r;
        return cudaGetLastError() == cudaSuccess ? EEMD_SP_OK : EEMD_SP_E_CUDA;
    }
    // the caller's rows stay untouched: the transform runs on complex copies
    k_promote<<<grid_for(total), 256, 0, st>>>(x, b.x, total);
    double2* spec = fft_rows(b.x, b.y, b.z, b.extra, M, L.P, -1, st);
    k_analytic<<<grid_for(total), 256, 0, st>>>(spec, b.x, M, N);
    double2* z = fft_rows(b.x, b.y, b.z, b.extra, M, L.P, +1, st);
    k_if_amp<<<grid_for(total), 256, 0, st>>>(z, inst_freq, inst_amp, M, N, sr);
    return cudaGetLastError() == cudaSuccess ? EEMD_SP_OK : EEMD_SP_E_CUDA;
}

int32_t eemd_sp_stft_shape(int64_t N, int32_t nperseg, int32_t noverlap, int32_t* F, int32_t* T) {
    if (!F || !T) return EEMD_SP_E_BADARG;
    int f = 0, t = 0;
    const int rc = stft_shape(N, nperseg, noverlap, f, t);
    if (rc) return rc;
    *F = f;
    *T = t;
    return EEMD_SP_OK;
}

int32_t eemd_sp_stft_workspace(int32_t M, int64_t N, int32_t nperseg, int32_t noverlap, size_t* bytes) {
    if (!bytes || M < 1) return EEMD_SP_E_BADARG;
    int F = 0, T = 0;
    int rc = stft_shape(N, nperseg, noverlap, F, T);
    if (rc) return rc;
    FftLayout L;
    rc = fft_layout((int64_t)M * T, nperseg, L);
    if (rc) return rc;
    *bytes = L.total;
    return EEMD_SP_OK;
}

int32_t eemd_sp_stft(const double* x, int32_t M, int64_t N, int32_t nperseg, int32_t noverlap, double* Z, void* ws,
                     size_t ws_bytes, void* stream) {
    if (!x || !Z || !ws || M < 1) return EEMD_SP_E_BADARG;
    int F = 0, T = 0;
    int rc = stft_shape(N, nperseg, noverlap, F, T);
    if (rc) return rc;
    FftLayout L;
    rc = fft_layout((int64_t)M * T, nperseg, L);
    if (rc) return rc;
    if (ws_bytes < L.total) return EEMD_SP_E_NOMEM;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Bufs b = carve(ws, L);
    const double wsum = window_sum(nperseg);
    StftPlan S;
    if (stft_plan(nperseg, M, nperseg - noverlap, T, S)) {
        const int64_t blocks = (int64_t)M * ((T + S.fb - 1) / S.fb);
        const int P = blocks <= FEW_CTAS && fft_threads(S.p, S.fb, 8) <= FFT_THREADS ? 8 : 16;
        const auto fn = nperseg % 2 ? (P == 8 ? k_stft<false, 8> : k_stft<false, 16>)
                                    : (P == 8 ? k_stft<true, 8> : k_stft<true, 16>);
        if (!smem_ready(reinterpret_cast<const void*>(fn))) return EEMD_SP_E_CUDA;
        const size_t sm = (size_t)(S.fb + 1) * pad8(S.p.n + 8) * sizeof(double2);
        const int nt = fft_threads(S.p, S.fb, P);
        fn<<<persistent_grid(blocks, nt, sm), nt, sm, st>>>(x, reinterpret_cast<double2*>(Z), M, N,
                                                                            1.0 / wsum, S);
        return cudaGetLastError() == cudaSuccess ? EEMD_SP_OK : EEMD_SP_E_CUDA;
    }
    k_frames<<<grid_for((int64_t)M * T * nperseg), 256, 0, st>>>(x, b.x, M, N, nperseg, nperseg - noverlap, T);
    double2* spec = fft_rows(b.x, b.y, b.z, b.extra, M * T, L.P, -1, st);
    k_stft_out<<<grid_for((int64_t)M * F * T), 256, 0, st>>>(spec, reinterpret_cast<double2*>(Z), M, F, T, nperseg,
                                                             1.0 / wsum);
    return cudaGetLastError() == cudaSuccess ? EEMD_SP_OK : EEMD_SP_E_CUDA;
}

}  // extern "C"
