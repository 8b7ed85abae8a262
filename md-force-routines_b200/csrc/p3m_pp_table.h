// FP64 pair table of the pair loop, built on the host (plain C++: a host test
// compiles this header too).
//
// psi(r) = phi(r) r = 1/2 [e^{kr} erfc(ar + c) + e^{-kr} erfc(ar - c)], c = k/2a
// (yukawa_pp.py:115), on [0, rc]: one polynomial of degree 7 per interval of h =
// rc / N, in u in [-1/2, 1/2] about its middle. The kernel takes the energy from
// psi and the force from g = F r^2 = psi - r psi' of the same polynomial.
//
// With G(r) = (2a / sqrt(pi)) e^{-a^2 r^2 - c^2}, from the derivatives of erfc,
//   psi' = k/2 [e^{kr} erfc(ar + c) - e^{-kr} erfc(ar - c)] - G,
//   psi'' = k^2 psi + 2 a^2 r G,   G' = -2 a^2 r G,
// so psi's Taylor series about an interval's middle follows by recurrence from
// psi, psi' and G there. They come from the closed form at every PP64_RESTART-th
// interval and from the next interval's series between (backwards, the direction
// in which psi grows and errors do not). 512 intervals take 0.2 ms on one core;
// with the closed form at every node of every interval 4.
#pragma once
#include <cmath>

namespace p3m {

// Intervals: the smallest power of two from PP64_MIN_N to PP64_MAX_N that meets
// PP64_LIMIT. alpha rc = 3.5 takes 512 for kappa up to a few alpha. The pair loop
// of 1e4 particles, rc 6, two lanes each: 52 us with 512 intervals, 53 with 1024
// (64 KB of shared memory a block), 170 with the direct terms.
constexpr int PP64_MIN_N = 128, PP64_MAX_N = 1024;
constexpr int PP64_COEF = 8;
// Error of psi and g of a pair, relative to themselves: a far pair's term is as
// accurate as a close one's, and more so than the direct terms, whose exponent
// alone rounds at a few 2^-53 (a r)^2.
constexpr double PP64_LIMIT = 4e-16;

constexpr int PP64_RESTART = 8;

// Coefficient q of interval i: the kernel reads pairs (2q, 2q + 1) as one 16-byte
// word, the pairs of all intervals together.
inline int pp64_at(int N, int i, int q) { return 2 * ((q / 2) * N + i) + q % 2; }

// What every interval uses: 1 / n, and the polynomials of degree K - 1 through
// u^n, n >= K, at the Chebyshev points of [-1/2, 1/2] (divided differences,
// expanded).
struct Pp64Constants {
    static constexpr int K = PP64_COEF, ORDER = 16;  // coefficients kept, Taylor terms
    long double inv[ORDER + 1], E[ORDER - K][K];
    Pp64Constants()
    {
        const long double pi = 3.141592653589793238462643383279502884L;
        long double x[K], f[K];
        for (int n = 1; n <= ORDER; ++n) inv[n] = 1.0L / n;
        for (int j = 0; j < K; ++j) x[j] = 0.5L * cosl((2 * j + 1) * pi / (2 * K));
        for (int n = K; n < ORDER; ++n) {
            long double *q = E[n - K];
            for (int j = 0; j < K; ++j) {
                f[j] = powl(x[j], n);
                q[j] = 0.0L;
            }
            for (int m = 1; m < K; ++m)
                for (int j = K - 1; j >= m; --j) f[j] = (f[j] - f[j - 1]) / (x[j] - x[j - m]);
            for (int m = K - 1; m >= 0; --m) {  // q = q (u - x[m]) + f[m]
                for (int j = K - 1; j > 0; --j) q[j] = q[j - 1] - x[m] * q[j];
                q[0] = f[m] - x[m] * q[0];
            }
        }
    }
};

// The table with N intervals, out[N * PP64_COEF]. Returns the largest relative
// error of psi and g, from the rounded coefficients, at each interval's ends and
// middle (the error of psi' is largest at the ends); stops at the first interval
// beyond `limit`. Intervals from the last on: there the limit fails first.
inline double build_pp_table64(double kappa, double alpha, double rc, int N, double limit, double *out)
{
    constexpr int K = PP64_COEF, ORDER = Pp64Constants::ORDER;
    const long double pi = 3.141592653589793238462643383279502884L;
    const long double k = kappa, a = alpha, c = 0.5L * k / a, h = (long double)rc / N, a2 = 2.0L * a * a;
    const long double h2 = h * h, a2h = -a2 * h;
    static const Pp64Constants C;
    // a series and its slope at u
    auto eval = [](const double *s, double u, double *slope) {
        double p = 0.0, d = 0.0;
        for (int n = ORDER - 1; n >= 0; --n) {
            d = d * u + p;
            p = p * u + s[n];
        }
        *slope = d;
        return p;
    };
    double worst = 0.0;
    long double G[ORDER], P[ORDER];  // Taylor coefficients in u = (r - middle) / h
    double Pd[ORDER], D[ORDER];      // psi's, and the table's less psi's
    for (int i = N - 1; i >= 0; --i) {
        const long double r = (i + 0.5L) * h;
        if ((N - 1 - i) % PP64_RESTART == 0) {
            const long double ekr = expl(k * r);
            const long double ep = ekr * erfcl(a * r + c), em = erfcl(a * r - c) / ekr;
            G[0] = 2.0L * a / sqrtl(pi) * expl(-a * a * r * r - c * c);
            P[0] = 0.5L * (ep + em);
            P[1] = h * (0.5L * k * (ep - em) - G[0]);
        } else {  // the next interval's series at its u = -1
            long double p = 0.0L, slope = 0.0L, g = 0.0L;
            for (int n = ORDER - 2; n >= 0; n -= 2) {
                p += P[n] - P[n + 1];
                slope += (n + 1) * P[n + 1] - n * P[n];
                g += G[n] - G[n + 1];
            }
            P[0] = p;
            P[1] = slope;
            G[0] = g;
        }
        for (int n = 0; n + 1 < ORDER; ++n) {
            const long double rG = r * G[n] + (n > 0 ? h * G[n - 1] : 0.0L);
            G[n + 1] = a2h * rG * C.inv[n + 1];
            if (n + 2 < ORDER) P[n + 2] = h2 * (k * k * P[n] + a2 * rG) * (C.inv[n + 1] * C.inv[n + 2]);
        }
        for (int j = 0; j < K; ++j) {
            long double q = P[j];
            for (int n = K + j % 2; n < ORDER; n += 2) q += P[n] * C.E[n - K][j];  // (the others are zero)
            out[pp64_at(N, i, j)] = (double)q;
        }
        for (int j = 0; j < ORDER; ++j) {
            Pd[j] = (double)P[j];
            D[j] = (double)(j < K ? out[pp64_at(N, i, j)] - P[j] : -P[j]);
        }
        for (int e = -1; e <= 1; ++e) {
            const double u = 0.5 * e, t = i + 0.5 + u;
            double slope, dslope;
            const double psi = eval(Pd, u, &slope), dpsi = eval(D, u, &dslope);
            const double err = fmax(fabs(dpsi / psi), fabs((dpsi - t * dslope) / (psi - t * slope)));
            if (!(err <= limit)) return HUGE_VAL;
            worst = fmax(worst, err);
        }
    }
    return worst;
}

}  // namespace p3m
