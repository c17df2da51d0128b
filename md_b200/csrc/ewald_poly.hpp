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
// truncated Chebyshev series in long double, turned into powers of u (their
// magnitudes sum to about 1.3 times the largest value).  In double the error is
// 2-5e-16 of the largest value of P or Q, everywhere: near the cutoff, where
// erfc(x)/r has fallen to 1e-7 of 1/r, that is 1e-9 of the term itself, and
// 1e-16 of the terms of near pairs that it is added to.
// A fit takes 0.04 ms of the host (1.0 ms with a cosine evaluated per product).
#pragma once

#include <cmath>
#include <vector>

namespace mdf {

constexpr int EWALD_DEG = 26;
constexpr double EWALD_Z_MAX = 13.3;   // ewald_tol >= 1e-6 has Z <= 13.13

// P and Q at z: power series below z = 2, the closed forms above.
inline void ewald_pq(long double z, long double& P, long double& Q)
{
    const long double spi = sqrtl(acosl(-1.0L));
    if (z < 2.0L) {
        long double t = 1.0L, s = 0.0L, u = 0.0L;
        for (int k = 0; k < 40 && fabsl(t) > 1e-24L; ++k) {
            s += t / (2 * k + 1);
            u += t / (2 * k + 3);
            t *= -z / (k + 1);
        }
        P = s * 2.0L / spi;
        Q = u * 4.0L / spi;
        return;
    }
    const long double x = sqrtl(z), e = erfl(x);
    P = e / x;
    Q = (e - 2.0L * x / spi * expl(-z)) / (x * z);
}

inline long double ewald_p(long double z)
{
    long double p, q;
    ewald_pq(z, p, q);
    return p;
}

inline long double ewald_q(long double z)
{
    long double p, q;
    ewald_pq(z, p, q);
    return q;
}

// Chebyshev nodes of the fit, and cos(pi m / (2 M)) over a whole turn: what the
// fit multiplies by, made once.  48 nodes take the coefficients above degree 69
// for those of degrees up to 26, far below the rounding.
constexpr int EWALD_NODES = 48;

inline const long double* ewald_cosines()
{
    static const std::vector<long double> c = [] {
        std::vector<long double> v(4 * EWALD_NODES);
        const long double pi = acosl(-1.0L);
        for (int m = 0; m <= EWALD_NODES; ++m) {
            const long double w = m == EWALD_NODES ? 0.0L : cosl(pi * m / (2 * EWALD_NODES));
            v[m] = w;
            v[2 * EWALD_NODES - m] = -w;
            v[(2 * EWALD_NODES + m) % (4 * EWALD_NODES)] = -w;
            v[(4 * EWALD_NODES - m) % (4 * EWALD_NODES)] = w;
        }
        v[0] = 1.0L;
        v[2 * EWALD_NODES] = -1.0L;
        return v;
    }();
    return c.data();
}

// Coefficients of u^0 .. u^EWALD_DEG, u = 2 z/Z - 1, from the values v at the nodes.
inline void ewald_fit(const long double* v, long double scale, double* out)
{
    const int M = EWALD_NODES, D = EWALD_DEG;
    const long double* cs = ewald_cosines();
    long double c[D + 1] = {}, t0[D + 1] = {}, t1[D + 1] = {}, t2[D + 1];
    t0[0] = 1.0L;   // T_0
    t1[1] = 1.0L;   // T_1
    for (int n = 0; n <= D; ++n) {
        long double b = 0.0L;
        for (int k = 0, m = n; k < M; ++k, m = (m + 2 * n) % (4 * M)) b += v[k] * cs[m];   // cos(pi n (k + 1/2) / M)
        b *= (n ? 2.0L : 1.0L) / M;
        for (int j = n & 1; j <= n; j += 2) c[j] += b * t0[j];   // T_n has the powers of n's parity
        for (int j = 0; j <= D; ++j) t2[j] = (j ? 2.0L * t1[j - 1] : 0.0L) - t0[j];
        for (int j = 0; j <= D; ++j) {
            t0[j] = t1[j];
            t1[j] = t2[j];
        }
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
    long double vp[EWALD_NODES], vq[EWALD_NODES];
    for (int k = 0; k < EWALD_NODES; ++k) ewald_pq(0.5L * Z * (1.0L + ewald_cosines()[2 * k + 1]), vp[k], vq[k]);
    ewald_fit(vp, a, t.p);
    ewald_fit(vq, a * a * a, t.q);
    t.on = 1;
    return t;
}

}  // namespace mdf
