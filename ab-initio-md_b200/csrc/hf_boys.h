// The Boys function F_N from a table: its layout, how it is made (host) and how
// it is read (device; the host too, so that it can be tested there).
//
// Below x = 36 + 3N one interval of width 1/8 gives F_N as a polynomial of
// degree 7 in the distance d from its middle c (interpolated at the Chebyshev
// nodes in extended precision), and e^-x = e^-c e^-d with e^-d by its Taylor
// series to d^8 (|d| <= 1/16); the lower orders follow by the downward
// recursion. From 36 + 3N on, F_n = (2n - 1)!! / (2x)^n F_0 with
// F_0 = sqrt(pi / x) / 2 holds to 1e-16 (the neglected part is of order
// x^(N - 1/2) e^-x / Gamma(N + 1/2)). Nine loads and some 25 operations, where
// the series and erf branches of boys_top take 50 and 150 and a warp that holds
// both kinds of x pays for both. The table of one order (9 coefficient columns of
// 288 + 24N rows, 21 to 31 KB) is staged in shared memory: the rows of a warp's
// lanes are scattered, which columns of coefficients spread over the banks.
// Largest relative error over all orders and x <= 300 (mean): N = 4 8.9e-16
// (1.0e-16) against 1.0e-15 (1.8e-16) of the branches, N = 6 8.9e-16 (1.1e-16). One B200,
// branches -> table: (H2O)32 J/K 118 -> 106 ms and gradient 176 -> 160 ms,
// (H2O)8 difference build 4.2 -> 3.5 ms.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#ifdef __CUDACC__
#define AIMD_HD __host__ __device__
#define AIMD_HD_INLINE __host__ __device__ __forceinline__
#else
#define AIMD_HD
#define AIMD_HD_INLINE inline
#endif

namespace hf {

// The highest order that a kernel reads: dd|ds, dd|pp and dp|dp in J/K.
constexpr int BOYS_MAX_N = 6, BOYS_COLS = 9;
AIMD_HD constexpr int boys_rows(int N) { return 8 * (36 + 3 * N); }
AIMD_HD constexpr int boys_offset(int N) {      // first element of order N in the table of all orders
    int o = 0;
    for (int m = 0; m < N; ++m) o += BOYS_COLS * boys_rows(m);
    return o;
}

// The tables of orders 0 .. BOYS_MAX_N: per interval the polynomial in d = x - c
// that interpolates F_N at the eight Chebyshev nodes, and e^-c. F_N at a node:
// the ascending series of the top order in extended precision, then the
// downward recursion.
inline std::vector<double> make_boys_tables() {
    constexpr int K = BOYS_COLS - 1, M = BOYS_MAX_N;
    const long double pi = 3.14159265358979323846264338327950288L, half = 1.0L / 16;    // half the interval
    std::vector<double> out(boys_offset(M + 1));
    long double node[4 * K];                        // cos(pi m / 2K)
    for (int m = 0; m < 4 * K; ++m) node[m] = cosl(pi * m / (2 * K));
    // monomial coefficients of the Chebyshev polynomials T_j
    long double tc[K][K] = {};
    tc[0][0] = tc[1][1] = 1.0L;
    for (int j = 2; j < K; ++j)
        for (int k = 0; k <= j; ++k) tc[j][k] = (k > 0 ? 2.0L * tc[j - 1][k - 1] : 0.0L) - tc[j - 2][k];
    for (int i = 0; i < boys_rows(M); ++i) {
        const long double c = (i + 0.5L) / 8;
        long double f[M + 1][K];
        for (int k = 0; k < K; ++k) {
            const long double x = c + half * node[2 * k + 1], ex = expl(-x);
            long double term = 1.0L / (2 * M + 1), sum = term;
            for (int n = 1; term > 1e-22L * sum; ++n) sum += term *= 2.0L * x / (2 * M + 2 * n + 1);
            f[M][k] = ex * sum;
            for (int n = M - 1; n >= 0; --n) f[n][k] = (2.0L * x * f[n + 1][k] + ex) / (2 * n + 1);
        }
        for (int n = 0; n <= M; ++n) {
            const int rows = boys_rows(n);
            if (i >= rows) continue;
            long double mono[K] = {};
            for (int j = 0; j < K; ++j) {
                long double a = 0.0L;
                for (int k = 0; k < K; ++k) a += f[n][k] * node[j * (2 * k + 1) % (4 * K)];
                a *= (j == 0 ? 1.0L : 2.0L) / K;
                for (int k = 0; k <= j; ++k) mono[k] += a * tc[j][k];
            }
            double* t = out.data() + boys_offset(n) + i;
            long double s = 1.0L;
            for (int k = 0; k < K; ++k, s /= half) t[k * rows] = static_cast<double>(mono[k] * s);
            t[K * rows] = static_cast<double>(expl(-c));
        }
    }
    return out;
}

AIMD_HD_INLINE int low_word(double x) {
#ifdef __CUDA_ARCH__
    return __double2loint(x);
#else
    int64_t b;
    memcpy(&b, &x, sizeof b);
    return static_cast<int>(b);
#endif
}
AIMD_HD_INLINE double inv_sqrt(double x) {
#ifdef __CUDA_ARCH__
    return rsqrt(x);
#else
    return 1.0 / sqrt(x);
#endif
}

// g[n] = scale (-2 alpha)^n F_n(T), n = 0..L, from the table t of order L
struct BoysShared {
    const double* t;
    template <int L>
    AIMD_HD_INLINE void operator()(double alpha, double T, double scale, double (&g)[L + 1]) const {
        constexpr int NR = boys_rows(L);
        if (!(T < 36 + 3 * L)) {        // (NaN too)
            const double r = inv_sqrt(T);
            double s = r * r;
            s = fma(s, fma(-T, s, 1.0), s) * -alpha;        // 1 / T to rounding (one Newton step)
            g[0] = 0.88622692545275801365 * r * scale;
#pragma unroll
            for (int n = 1; n <= L; ++n) g[n] = g[n - 1] * ((2 * n - 1) * s);
            return;
        }
        // row floor(8 T), as the integer nearest to 8 T - 1/2: adding 1.5 2^52
        // leaves it in the low word (no conversion instructions)
        const double m = fma(T, 8.0, -0.5) + 6755399441055744.0;
        const double d = fma(-0.125, m - 6755399441055744.0, T - 0.0625);
        const double* c = t + low_word(m);
        double f = c[7 * NR];
#pragma unroll
        for (int j = 6; j >= 0; --j) f = fma(f, d, c[j * NR]);
        if constexpr (L == 0) {
            g[0] = f * scale;
        } else {
            double e = 1.0 / 40320;
            e = fma(e, d, -1.0 / 5040);
            e = fma(e, d, 1.0 / 720);
            e = fma(e, d, -1.0 / 120);
            e = fma(e, d, 1.0 / 24);
            e = fma(e, d, -1.0 / 6);
            e = fma(e, d, 0.5);
            e = fma(e, d, -1.0);
            const double e0 = c[8 * NR], ex = fma(e * d, e0, e0);
            const double m2a = -2.0 * alpha, T2 = 2.0 * T;
            double pw[L + 1];
            pw[0] = scale;
#pragma unroll
            for (int n = 1; n <= L; ++n) pw[n] = pw[n - 1] * m2a;
            g[L] = pw[L] * f;
#pragma unroll
            for (int n = L - 1; n >= 0; --n) {
                f = fma(T2, f, ex) * (1.0 / (2 * n + 1));
                g[n] = pw[n] * f;
            }
        }
    }
};

}  // namespace hf
