// Prints, for one alpha and cutoff, erfc(alpha r)/r and its force factor at n
// distances from the polynomials of md_b200/csrc/ewald_poly.hpp, evaluated in
// double by Horner's rule as the FP64 pair kernel does, and from the long
// double functions.
#include <cstdio>
#include <cstdlib>

#include "ewald_poly.hpp"

int main(int argc, char** argv)
{
    const double alpha = atof(argv[1]), rc = atof(argv[2]);
    const int n = atoi(argv[3]);
    const mdf::EwaldPoly t = mdf::make_ewald_poly(alpha, rc);
    if (!t.on) {
        printf("none\n");
        return 0;
    }
    for (int i = 0; i <= n; ++i) {
        const double r = rc * i / n, u = std::fma(r * r, 2.0 / (rc * rc), -1.0);
        double p = t.p[mdf::EWALD_DEG], q = t.q[mdf::EWALD_DEG];
        for (int k = mdf::EWALD_DEG - 1; k >= 0; --k) {
            p = std::fma(p, u, t.p[k]);
            q = std::fma(q, u, t.q[k]);
        }
        const long double a = alpha, z = a * a * (long double)r * r;
        printf("%.17g %.21Lg %.17g %.21Lg\n", p, a * mdf::ewald_p(z), q, a * a * a * mdf::ewald_q(z));
    }
    return 0;
}
