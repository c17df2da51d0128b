// Polynomials of the FP64 real-space Ewald terms (host code, no CUDA).
//
// With x = alpha r, z = x^2:
//   erfc(x) / r                                  = 1/r   - alpha   P(z)
//   (erfc(x)/r + 2 alpha/sqrt(pi) e^{-z}) / r^2  = 1/r^3 - alpha^3 Q(z)
//   P(z) = erf(x)/x = 2/sqrt(pi) int_0^1 e^{-z t^2} dt
//   Q(z) = (erf(x) - 2x/sqrt(pi) e^{-z}) / x^3 = 4/sqrt(pi) int_0^1 t^2 e^{-z t^2} dt
// P and Q are entire in z, so over the pairs inside the cutoff (z from 0 to
// Z = (alpha rc)^2) one polynomial of degree EWALD_DEG in u = 2 r^2/rc^2 - 1
// gives each to rounding: the Chebyshev coefficients fall like I_n(Z/2) e^{-Z/2},
// below 2e-17 at degree 27 for Z = EWALD_Z_MAX.  The coefficients are the
// truncated Chebyshev series in long double, turned into powers of u (all of
// them O(1), so Horner's rule loses nothing).
#pragma once

#include <cmath>
#include <vector>

namespace mdf {

constexpr int EWALD_DEG = 26;
constexpr double EWALD_Z_MAX = 13.3;   // ewald_tol >= 1e-6 has Z <= 13.13

inline long double ewald_p(long double z)
{
    if (z < 2.0L) {
        long double t = 1.0L, s = 0.0L;
        for (int k = 0; k < 40; ++k) {
            s += t / (2 * k + 1);
            t *= -z / (k + 1);
        }
        return s * 2.0L / sqrtl(acosl(-1.0L));
    }
    const long double x = sqrtl(z);
    return erfl(x) / x;
}

inline long double ewald_q(long double z)
{
    const long double spi = sqrtl(acosl(-1.0L));
    if (z < 2.0L) {
        long double t = 1.0L, s = 0.0L;
        for (int k = 0; k < 40; ++k) {
            s += t / (2 * k + 3);
            t *= -z / (k + 1);
        }
        return s * 4.0L / spi;
    }
    const long double x = sqrtl(z);
    return (erfl(x) - 2.0L * x / spi * expl(-z)) / (x * z);
}

// Coefficients of u^0 .. u^EWALD_DEG of f over z in [0, Z], u = 2 z/Z - 1.
template <typename F>
inline void ewald_fit(F f, long double Z, long double scale, double* out)
{
    const int M = 96, D = EWALD_DEG;
    const long double pi = acosl(-1.0L);
    std::vector<long double> v(M), b(D + 1), c(D + 1, 0.0L), t0(D + 1, 0.0L), t1(D + 1, 0.0L), t2(D + 1);
    for (int k = 0; k < M; ++k) v[k] = f(0.5L * Z * (1.0L + cosl(pi * (k + 0.5L) / M)));
    for (int n = 0; n <= D; ++n) {
        long double s = 0.0L;
        for (int k = 0; k < M; ++k) s += v[k] * cosl(pi * n * (k + 0.5L) / M);
        b[n] = s * (n ? 2.0L : 1.0L) / M;
    }
    t0[0] = 1.0L;   // T_0
    t1[1] = 1.0L;   // T_1
    for (int n = 0; n <= D; ++n) {
        for (int j = 0; j <= D; ++j) c[j] += b[n] * t0[j];
        for (int j = 0; j <= D; ++j) t2[j] = (j ? 2.0L * t1[j - 1] : 0.0L) - t0[j];
        t0 = t1;
        t1 = t2;
    }
    for (int j = 0; j <= D; ++j) out[j] = (double)(scale * c[j]);
}

// p, q: the coefficients of alpha P and alpha^3 Q; on = 0: none at this alpha
// and cutoff (alpha rc too large).
struct EwaldPoly {
    long long on;   // 64 bits: no padding, so tables compare by memory
    double p[EWALD_DEG + 1], q[EWALD_DEG + 1];
};

inline EwaldPoly make_ewald_poly(double alpha, double rc)
{
    EwaldPoly t{};
    const long double a = alpha, Z = a * a * (long double)rc * rc;
    if (!(Z <= (long double)EWALD_Z_MAX)) return t;
    ewald_fit(ewald_p, Z, a, t.p);
    ewald_fit(ewald_q, Z, a * a * a, t.q);
    t.on = 1;
    return t;
}

}  // namespace mdf
