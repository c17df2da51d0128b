// Launch arguments of the evaluation kernels, one struct per kernel.
//
// Every kernel of an evaluation takes its arguments as one struct, so the same
// body serves two launch forms:
//   k_X(XArgs a)                 one system, the struct passed by value;
//   k_X_multi(const XArgs* as)   many systems in one launch: blockIdx.z picks
//                                the system's struct in device memory, and
//                                blocks past that system's own grid (gx, gy)
//                                return at once.
// A system's blocks run the same code on the same data in both forms, so a
// batch launch reproduces the single-system results bit for bit (energies
// included: each block, or each i cluster in the persistent pair kernels,
// sums the same terms in the same order).
#pragma once

#include "mdf_device.cuh"
#include "mdf_internal.cuh"
#include "nb_common.cuh"

namespace mdf {

// The blocks of a many-system launch: a one-dimensional grid of n blocks,
// block b running block map[b].y (linear in the system's own gx x gy grid)
// of system map[b].x.
struct BlockMap {
    const int2* map;
    int n;
};

// ---------------------------------------------------------------- pairlist
template <typename R>
struct PackArgs {
    int gx, gy;
    int nslots;
    const double* xyz;
    const double* q;
    const int* slot_atom;
    const double4* center;
    double L[3];
    typename V4<R>::type* xq;
    float4* box;                        // current boxes (box_encode)
    float box_pad;
    float4* xf;                         // FP64: the FP32 copy of xq
    const typename V4<R>::type* snap;   // self-pruning: positions of the last prune (nullptr: off)
    unsigned* disp;                     // largest squared displacement from snap (FP32 bits, atomicMax)
    unsigned* st;
};

struct PruneArgs {
    int gx, gy;
    int ncl;
    int warps;              // warps per i cluster: 1 or 4
    const ILRange* ilist;
    const PairEntry* plist;
    const float4* xf;
    const double4* xd;      // FP64 contexts: the offsets in FP64 (snap_d, wide clusters); mixed: null
    const float4 *centerf, *box;
    int box_fine;           // box padding small enough for the acceptance by boxes
    ShiftTable shifts;
    float rcut2;
    ILRange* ilist_in;
    PairEntry* plist_in;
    // self-pruning: prune only when force is set or the displacement since the
    // last prune (written by the pack kernel) exceeds disp_thr2; a prune that
    // runs records the positions it used in the snapshot of the precision
    float4* snap_f;
    double4* snap_d;
    const unsigned* disp;
    float disp_thr2;
    int force;
};

// Launch on the context's present stream of a kernel that runs beside its pair
// kernel, asking for an L1 divided as the pair kernel divides it: 72% shared
// memory with blocks of eight warps, all of it with smaller ones.  An SM has to
// drain to change the division, and left to itself a kernel that needs little
// shared memory gets little: where the pair kernel's blocks all fit on the chip at
// once, the side streams' kernels then wait for it to end.  Unpruned mixed
// evaluations back to back (with energies / forces alone): 20,400 atoms 168 / 205
// us with the driver's choice, 140 / 145 with this; 27,600 179 / 216 and 139 / 159;
// 100k pruned, two evaluations, 668 and 648; FP64 at 20,400 188 and 175; 2,800 the
// same.  72% beside blocks of two or four warps costs 5-25%, 100% beside eight-warp
// ones 1.5% from 100k atoms on.  A batch keeps the driver's choice (128 systems
// 3.30 ms, 3.38 with 72%, 3.49 with 100%).
template <typename... P, typename... A>
void launch_beside(const Ctx& c, void (*kern)(P...), dim3 grid, int threads, size_t smem, A&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = c.p.pair_warps == 2 || c.p.pair_warps == 4 ? 100 : 72;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    MDF_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
}

// ------------------------------------------------------------- pair kernels
constexpr int WHOLE_LIST = 1 << 30;   // a list is one part (PairF32Args::part)

// Constants of the FP32 pair kernel, folded on the host.
struct PairConstF {
    float rc2;
    float kex;        // -alpha^2 log2(e): exp(-alpha^2 r^2) = 2^(kex r^2)
    float pa;         // 0.3275911 alpha (A&S 7.1.26 argument)
    float two_a_spi;  // 2 alpha / sqrt(pi)
    float inv_sw, rsw_inv;          // 1/(rc - rsw), rsw/(rc - rsw)
    float d30, d60;                 // -30, 60 times inv_sw (dS/dr = x^2 (d30 + x (d60 + x d30)))
    float uc6, uc12, rcf, rc2f;     // force-shifted LJ
};

struct PairF32Args {
    int gx, gy;
    int nlist;
    const ILRange* ilist;
    const PairEntry* plist;
    const float4* xq;
    const int* stype;
    const float4* centerf;
    const float4* lj4;
    int ntp;
    int lj_smem;
    float kc;
    PairConstF K;
    ShiftTable shifts;
    unsigned long long* fslot;
    int nslots;
    unsigned long long* acc;
    unsigned long long* npairs;
    unsigned long long* next;   // work counter of the persistent warps, zero at launch
    int persist;                // 1: persistent warps on the counter; 0: warp w takes item w
    int half;                   // lists are half entries (the 4 x 8 kernel)
    int split;                  // log2 of the shares (items) each list is cut into
    int part;                   // entries per part (pair_part), or WHOLE_LIST
    unsigned* st;
};

// Constants and image offsets of the FP64 PHYSICAL pair kernel (the same
// structure as the FP32 kernel's, in double).
struct PairConstD {
    double rc2, alpha, two_a_spi;
    double inv_sw, rsw_inv, d30, d60;   // switch: x = r inv_sw - rsw_inv; dS/dr = x^2 (d30 + x (d60 + x d30))
    double uc6, uc12, rc;               // force-shifted LJ
    double two_rc2;                     // 2 / rc^2 (argument of the Ewald polynomials)
};

struct ShiftTableD {
    double v[27][3];
};

struct PairF64Args {
    int gx, gy;
    int nlist;
    const ILRange* ilist;
    const PairEntry* plist;
    const double4* xq;
    const int* stype;
    const double4* center;
    const double4* lj4;     // (A, B, 12A, 6B) per type pair
    int ntp;
    int lj_smem;
    double kc;
    PairConstD K;
    ShiftTableD shifts;
    unsigned long long* fslot;
    int nslots;
    unsigned long long* acc;
    unsigned long long* npairs;
    unsigned long long* next;   // work counter of the persistent warps, zero at launch
    int persist;                // 1: persistent warps on the counter; 0: warp w takes item w
    int half;                   // lists are half entries (the 4 x 8 kernel)
    EwaldPoly poly;
    unsigned* st;
};

// The FP64 real-space Ewald terms of a pair per q_i q_j: energy erfc(alpha r)/r
// and the force factor (that + 2 alpha/sqrt(pi) e^{-alpha^2 r^2})/r^2.
//
// What bounds the FP64 kernels is the double-precision pipe (a warp
// instruction takes it two cycles), and exp and erfc were more than half of
// what a pair put on it.  Over the cutoff's range both terms are 1/r and 1/r^3
// minus one polynomial each in r^2 (ewald_poly.hpp; 2-5e-16 of the largest
// value): 52 FMAs instead of exp + erfc, 26 when only forces are wanted, and
// coefficients that the FMA reads from the constant bank.  Slots outside the
// cutoff, padding and an atom with itself give any value, infinities and NaN
// among them: the caller selects them away and must not multiply them by zero.
// With an alpha rc beyond EWALD_Z_MAX (ewald_tol below 1e-6) the functions
// themselves are called.  Pair launch at 100k atoms (half lists, energies)
// 572 -> 392 us, forces alone 555 -> 330; 28k atoms 251 -> 155; 7,309 atoms
// 178 -> 113; a batch of 64 small systems 1.92 -> 1.39 ms.
template <bool POLY, bool ENERGY>
__device__ __forceinline__ void ewald_f64(const EwaldPoly& T, const PairConstD& K, double r2, double r,
                                          double rinv, double rinv2, double& e, double& f)
{
    if (POLY) {
        const double u = fma(r2, K.two_rc2, -1.0);
        double P = T.p[EWALD_DEG], Q = T.q[EWALD_DEG];
#pragma unroll
        for (int k = EWALD_DEG - 1; k >= 0; --k) {
            if (ENERGY) P = fma(P, u, T.p[k]);
            Q = fma(Q, u, T.q[k]);
        }
        e = ENERGY ? rinv - P : 0.0;
        f = fma(rinv, rinv2, -Q);
    } else {
        const double ar = K.alpha * r;
        e = erfc(ar) * rinv;
        f = fma(K.two_a_spi, exp(-ar * ar), e) * rinv2;
    }
}

template <typename R>
struct PairArgs {
    int gx, gy;
    int nlist;
    const ILRange* ilist;
    const PairEntry* plist;
    const typename V4<R>::type* xq;
    const int* stype;
    const double4* center;
    const typename V2<R>::type* ljAB;
    const int* ljvalid;
    NBParams P;
    unsigned long long* fslot;
    int nslots;
    unsigned long long* acc;
    unsigned long long* npairs;
    int count;
    unsigned* st;
};

struct ExclArgs {
    int gx, gy;
    int n;
    const int* pairs;
    const int* is14;
    const double* xyz;
    const double* q;
    NBParams P;
    int N;
    unsigned long long* fatom;
    unsigned long long* acc;
    unsigned* st;
};

struct Pair14Args {
    int gx, gy;
    int n;
    const int* pairs;
    const double2* scale;
    const double* xyz;
    const double* q;
    const int* type;
    const double2* lj14;
    const int* ljvalid;
    NBParams P;
    int N;
    unsigned long long* fatom;
    unsigned long long* acc;
    unsigned* st;
};

// ------------------------------------------------------------------ bonded
struct BondedArgs {
    int gx, gy;
    int n[6];        // end index per list: bonds, ub, angles, dihedrals, impropers, cmaps
    int lo[6];       // first index per list (a rank's share starts there)
    int blk0[7];     // first block of each segment (prefix)
    const int *bond_atoms, *ub_atoms, *angle_atoms, *dih_atoms, *imp_atoms, *cmap_atoms, *cmap_set;
    const double2 *bond_par, *ub_par, *angle_par, *imp_par;
    const double* dih_par;
    const double* cmap_coeff;
    int cmap_res;
    const double* xyz;
    int N;
    unsigned long long* f;
    unsigned long long* acc;
    unsigned* st;
};

// Bonded terms, excluded pairs and 1-4 pairs of one system (gx = the sum of
// their blocks; a part left out has gx = 0).
struct TermArgs {
    int gx, gy;
    BondedArgs b;
    ExclArgs e;
    Pair14Args p;
};

// --------------------------------------------------------------------- PME
struct GridGeom {
    int K[3];
    double L[3];
    double scale[3];   // K/L
};

struct FFTDesc {
    int n;
    int nst;
    int radix[12];
    int ns[12];
    int toff[12];
    int ntab;
    int r[3];         // register radices (fft_regs.cuh); r[0] = 0: none, the table-driven passes
};

struct ConvParams {
    int K[3];
    double pa2;       // pi^2 / alpha^2 (virial factor)
    int reference;    // REFERENCE solve: no energy or virial
};

struct ZeroArgs {
    int gx, gy;
    unsigned long long* p;
    long long n;
};

struct SpreadArgs {
    int gx, gy;
    int s0, s1;
    const int* slot_atom;
    const double* xyz;
    const double* q;
    GridGeom g;
    unsigned long long* qgrid;
    unsigned* st;
    int win_lo, win_n;   // halo exchange: stencil bases must lie in win_lo .. +win_n-1 (mod K0); win_n = 0: any
};

template <typename R>
struct GatherArgs {
    int gx, gy;
    int s0, s1, nslots;
    const int* slot_atom;
    const double* xyz;
    const double* q;
    GridGeom g;
    const R* phi;
    unsigned long long* fslot;
    unsigned* st;
};

// z passes (r2c: charge grid -> half complex; c2r: half complex -> potential).
// A launch of gridDim.z = 2 transforms a second set of grids beside the first
// (the adjoint's dipole chain); unused otherwise.
template <typename R>
struct FFTZArgs {
    int gx, gy;
    const unsigned long long* qgrid;              // r2c input
    typename V2<R>::type* cgrid;                   // r2c output / c2r input
    R* rgrid;                                      // c2r output
    const unsigned long long* qgrid2;              // the second set
    typename V2<R>::type* cgrid2;
    R* rgrid2;
    int nlines;
    FFTDesc d;
    const typename V2<R>::type* tw;
    const int2* tab;
    int LP;
};

template <typename R>
struct FFTYArgs {
    int gx, gy;
    typename V2<R>::type *cgrid, *cgrid2;
    int Kc;
    FFTDesc d;
    const typename V2<R>::type* tw;
    const int2* tab;
    int LP, lp_shift;
    int inverse;
};

template <typename R>
struct FFTXArgs {
    int gx, gy;
    typename V2<R>::type *cgrid, *cgrid2;
    int K1, Kc;
    FFTDesc d;
    const typename V2<R>::type* tw;
    const int2* tab;
    int LP, lp_shift;
    ConvParams cp;
    const R* infl;
    const double *mx, *my, *mz;
    unsigned long long* acc;
    unsigned* st;
};

// One system's FFT chain: the five passes and their dynamic shared memory.
template <typename R>
struct FFTChain {
    FFTZArgs<R> zf, zi;
    FFTYArgs<R> yf, yi;
    FFTXArgs<R> x;
    size_t smz, smy, smx;
    bool energy;
};

// Many systems' chains: device arrays [nsys] of each pass's arguments ...
template <typename R>
struct FFTChainDev {
    const FFTZArgs<R>* zf;
    const FFTYArgs<R>* yf;
    const FFTXArgs<R>* x;
    const FFTYArgs<R>* yi;
    const FFTZArgs<R>* zi;
    // the blocks of the z, y and x passes (forward and inverse share them): [0] table-driven, [1] register radices
    BlockMap mz[2], my[2], mx[2];
};

// ... and the largest shared memory of each pass over the systems.
struct FFTChainMax {
    size_t smz[2], smy[2], smx[2];
};

// --------------------------------------------------------------- finalize
struct FinalizeArgs {
    int gx, gy;
    int N, nslots;
    unsigned long long* fatom;
    unsigned long long* fslot;
    const int* atom_slot;
    double* out;
    unsigned long long* scal;
    unsigned long long* host_scal;
};

// ----------------------------------------------------- host-side builders
// The arguments of one system's launch (from its context) and the
// many-system launchers (device arrays of arguments, the largest grid).
template <typename R> PackArgs<R> make_pack_args(const Ctx& c);
template <typename R> void launch_pack_multi(const PackArgs<R>* d_args, BlockMap bm, cudaStream_t s);
PruneArgs make_prune_args(const Ctx& c, bool half);
void set_prune_warps(PruneArgs& A, long long ncl);   // by the clusters of the whole launch
void ensure_half_lists(Ctx& c);
void launch_prune_multi(const PruneArgs* d_args, int nsys, int gx, int warps, bool half, bool wide, bool selfp,
                        cudaStream_t s);
PairF32Args make_pair_f32_args(const Ctx& c, size_t* dyn);
void launch_pairs_f32_multi(const PairF32Args* d_args, int nsys, int gx, int threads, size_t dyn, bool energy,
                            bool use_switch, bool persist, bool half, bool lj_smem, bool parts, cudaStream_t s);
template <typename R> PairArgs<R> make_pair_args(const Ctx& c, bool count);
PairF64Args make_pair_f64_args(const Ctx& c, size_t* dyn);
void launch_pairs_f64_multi(const PairF64Args* d_args, int nsys, int gx, int threads, size_t dyn, bool energy,
                            bool use_switch, bool persist, bool half, bool lj_smem, const EwaldPoly& poly, cudaStream_t s);
int pair_threads(const Ctx& c);
int pair_split(long long nlist);
// 2^split items per list, one warp each.
inline void set_pair_split(PairF32Args& a, int split, int warps_per_block)
{
    a.split = a.part < WHOLE_LIST ? split : 0;
    a.gx = grid_blocks((long long)a.nlist << a.split, warps_per_block);
}
ExclArgs make_excl_args(const Ctx& c);
Pair14Args make_pair14_args(const Ctx& c);
BondedArgs make_bonded_args(const Ctx& c, bool whole, unsigned long long* f, unsigned long long* acc, unsigned* st);
TermArgs make_term_args(const Ctx& c, bool energy, bool bonded, bool pairs);
void launch_terms_multi(const TermArgs* d_args, int nsys, int gx, bool energy, cudaStream_t s);
template <typename R> FFTChain<R> make_fft_chain(const Ctx& c, bool energy);
SpreadArgs make_spread_args(const Ctx& c);
template <typename R> GatherArgs<R> make_gather_args(const Ctx& c);
template <typename R>
void launch_pme_multi(const ZeroArgs* d_zero, BlockMap mzero, const SpreadArgs* d_spread, BlockMap mspread,
                      const FFTChainDev<R>& D, const FFTChainMax& M, const GatherArgs<R>* d_gather, BlockMap mgather,
                      bool energy, cudaStream_t s);
FinalizeArgs make_finalize_args(const Ctx& c, double* d_forces);
void launch_finalize_multi(const FinalizeArgs* d_args, BlockMap bm, cudaStream_t s);

// The grid of a one-system launch from the struct's own extents.
template <typename A>
inline dim3 grid_of(const A& a)
{
    return dim3((unsigned)a.gx, (unsigned)a.gy, 1u);
}

}  // namespace mdf
