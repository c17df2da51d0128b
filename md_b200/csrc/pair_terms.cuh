// Excluded pairs and 1-4 pairs in FP64 (block bodies; the kernel that runs them
// beside the bonded terms is in bonded.cu).
#pragma once

#include "kargs.cuh"
#include "mdf_device.cuh"
#include "nb_common.cuh"

namespace mdf {

// --------------------------------------------------------------- FP64 pairs
__device__ __forceinline__ void pair_vec(const double* __restrict__ xyz, int a, int b, const NBParams& P,
                                         double d[3])
{
    d[0] = min_image(xyz[3 * a] - xyz[3 * b], P.box[0]);
    d[1] = min_image(xyz[3 * a + 1] - xyz[3 * b + 1], P.box[1]);
    d[2] = min_image(xyz[3 * a + 2] - xyz[3 * b + 2], P.box[2]);
}

__device__ __forceinline__ void add_pair_force(unsigned long long* f, int N, int a, int b, double g, const double d[3],
                                               unsigned* st)
{
    for (int k = 0; k < 3; ++k) {
        fx_add(f + k * N + a, g * d[k], FORCE_SCALE, st);
        fx_add(f + k * N + b, -g * d[k], FORCE_SCALE, st);
    }
}

// Excluded pairs.  PHYSICAL: -k q q erf(alpha r)/r with its force (every
// excluded pair, min image, no cutoff).  REFERENCE: the same energy for
// excluded pairs that are not 1-4 (src/System/NonBondedEnergy.cpp:271-304),
// no force.
template <int SEM, bool ENERGY>
__device__ __forceinline__ void exclusions_dev(const ExclArgs& A, int bx)
{
    const int n = A.n;
    const int* __restrict__ pairs = A.pairs;
    const int* __restrict__ is14 = A.is14;
    const double* __restrict__ xyz = A.xyz;
    const double* __restrict__ q = A.q;
    const NBParams& P = A.P;
    const int N = A.N;
    unsigned long long* __restrict__ fatom = A.fatom;
    unsigned long long* __restrict__ acc = A.acc;
    unsigned* st = A.st;
    int k = bx * blockDim.x + threadIdx.x;
    double e = 0.0;
    if (k < n && !(SEM == MDF_SEM_REFERENCE && is14[k])) {
        int a = pairs[2 * k], b = pairs[2 * k + 1];
        double d[3];
        pair_vec(xyz, a, b, P, d);
        double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2], r = sqrt(r2);
        if (SEM == MDF_SEM_PHYSICAL) {
            double qq = q[a] * q[b] * P.kc, ar = P.alpha * r;
            e = -qq * erf(ar) / r;
            double g = (e + qq * (2.0 * P.alpha / 1.7724538509055160273) * exp(-ar * ar)) / r2;
            add_pair_force(fatom, N, a, b, g, d, st);
        } else {
            e = -P.kc * (q[a] * q[b] / r) * erf(P.alpha * r);
        }
    }
    if (ENERGY) {
        const double v[1] = {e};
        const int idx[1] = {SEM == MDF_SEM_PHYSICAL ? MDF_E_EE_EXCL : MDF_E_EE_DIRECT};
        block_acc_fixed<1>(v, acc, idx, ENERGY_SCALE, st);
    }
}

// 1-4 pairs.  PHYSICAL: k q q / (scee r) + (A14/r^12 - B14/r^6) / scnb.
// REFERENCE: the reference's is14 branches of the list loops (A14/B14 with the
// switch, Coulomb / scee, and CalculateEnergyEwaldDirectTerm_14's erf(r)).
template <int SEM, bool ENERGY>
__device__ __forceinline__ void pairs14_dev(const Pair14Args& A, int bx)
{
    const int n = A.n;
    const int* __restrict__ pairs = A.pairs;
    const double2* __restrict__ scale = A.scale;
    const double* __restrict__ xyz = A.xyz;
    const double* __restrict__ q = A.q;
    const int* __restrict__ type = A.type;
    const double2* __restrict__ lj14 = A.lj14;
    const int* __restrict__ ljvalid = A.ljvalid;
    const NBParams& P = A.P;
    const int N = A.N;
    unsigned long long* __restrict__ fatom = A.fatom;
    unsigned long long* __restrict__ acc = A.acc;
    unsigned* st = A.st;
    int k = bx * blockDim.x + threadIdx.x;
    double ev = 0, ec = 0, eall = 0, epl = 0, ecut = 0, edir = 0;
    if (k < n) {
        int a = pairs[2 * k], b = pairs[2 * k + 1];
        double d[3];
        pair_vec(xyz, a, b, P, d);
        double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2], r = sqrt(r2);
        double2 sc = scale[k];
        int tp = type[a] * P.ntp + type[b];
        double2 ab = lj14[tp];
        double i2 = 1.0 / r2, i4 = i2 * i2, i6 = i4 * i2, i8 = i4 * i4, i12 = i6 * i6, i14 = i12 * i2;
        if (SEM == MDF_SEM_PHYSICAL) {
            double qq = q[a] * q[b] * P.kc / sc.x;
            ec = qq / r;
            double g = ec / r2;
            if (ljvalid[tp]) {
                ev = (ab.x * i12 - ab.y * i6) / sc.y;
                g += (12.0 * ab.x * i14 - 6.0 * ab.y * i8) / sc.y;
            }
            add_pair_force(fatom, N, a, b, g, d, st);
        } else {
            double qq = q[a] * q[b];
            double scee = sc.x;
            if (r2 <= P.rc2 && r2 >= 1e-12) eall = (1.0 / scee) * ((qq / r) * P.kc);
            bool in_list = r2 <= P.rlist2 && r2 > 1e-12 && ljvalid[tp];
            if (in_list && r2 <= P.rc2 && r2 >= 1e-12) {
                double U = ab.x * i12 - ab.y * i6, G = 12.0 * ab.x * i14 - 6.0 * ab.y * i8;
                if (P.use_switch) {
                    double S = 1.0, dS = 0.0;
                    if (r > P.rsw) {
                        if (r >= P.rc) S = 0.0;
                        else {
                            double x = (r - P.rsw) * P.inv_sw, x2 = x * x, x3 = x2 * x, x4 = x2 * x2, x5 = x4 * x;
                            S = 1.0 - 10.0 * x3 + 15.0 * x4 - 6.0 * x5;
                            dS = (-30.0 * x2 + 60.0 * x3 - 30.0 * x4) * P.inv_sw;
                        }
                    }
                    G = S * G - (U / r) * dS;
                    U = U * S;
                } else {
                    double c2 = 1.0 / P.rc2, c4 = c2 * c2, c6 = c4 * c2, c8 = c4 * c4, c12 = c6 * c6, c14 = c12 * c2;
                    double ucut = ab.x * c12 - ab.y * c6, gcut = 12.0 * ab.x * c14 - 6.0 * ab.y * c8;
                    U = U - ucut + (r - P.rc) * (gcut * P.rc);
                    G = G - gcut * (P.rc / r);
                }
                ev = U;
                epl = (1.0 / scee) * ((qq / r) * P.kc);
                ecut = (1.0 / scee) * (qq * P.kc) * (1.0 / r - 1.0 / P.rc);
                edir = ((1.0 / (scee * r)) - (erf(r) / r)) * (qq * P.kc);
                double g = G + (1.0 / scee) * ((qq / (r2 * r)) * P.kc);
                add_pair_force(fatom, N, a, b, g, d, st);
            }
        }
    }
    if (ENERGY) {
        if (SEM == MDF_SEM_PHYSICAL) {
            const double v[2] = {ev, ec};
            const int idx[2] = {MDF_E_VDW14, MDF_E_EE14};
            block_acc_fixed<2>(v, acc, idx, ENERGY_SCALE, st);
        } else {
            const double v[5] = {ev, eall, epl, ecut, edir};
            const int idx[5] = {MDF_E_VDW, MDF_E_EE, MDF_E_EE_PAIRLIST, MDF_E_EE_CUTOFF, MDF_E_EE_DIRECT};
            block_acc_fixed<5>(v, acc, idx, ENERGY_SCALE, st);
        }
    }
}

}  // namespace mdf
