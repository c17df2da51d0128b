// Adjoint (vector-Jacobian product) of the PHYSICAL energy and forces with
// respect to the per-atom charges and the Lennard-Jones A/B coefficients.
//
// Given v = dL/dF (3N, forces as returned by mdf_compute) and gE = dL/dE
// (total energy), the gradient of the loss is the gradient, at fixed
// positions, of
//     Phi(q, A, B) = gE E + sum_a v_a . F_a .
// Every nonbonded pair contributes E_ab = A e_A(r) + B e_B(r) + q_a q_b e_0(r)
// and F_a = -F_b = g(r) d with g linear in the same coefficients, so per pair
//     dPhi/dA_ab = gE e_A + g_A w,   dPhi/dB_ab = gE e_B + g_B w,
//     dPhi/dq_a += q_b (gE e_0 + g_0 w),   w = (v_a - v_b) . d .
// The pair kernel is recomputed (nothing is stored by the forward pass).  The
// exclusion corrections, the 1-4 Coulomb pairs, the self energy and the net
// charge term follow the same pattern; the reciprocal space is in pme.cu.
//
// dL/dq is accumulated in int64 fixed point (deterministic); dL/dA and dL/dB
// per NONBONDED_PARM_INDEX entry in FP64 through per-block shared-memory
// partials (atomics in FP64: reproducible to rounding, not bitwise).
#include <algorithm>
#include <cmath>
#include <vector>

#include "kargs.cuh"
#include "mdf_device.cuh"
#include "mdf_internal.cuh"
#include "nb_common.cuh"

namespace mdf {

// dL/dq and the normalised v are scaled by 1/scale so that the fixed-point
// accumulators keep their resolution whatever the loss' magnitude.
template <typename R>
__global__ void k_adj_pack(int nslots, const int* __restrict__ slot_atom, const double* __restrict__ v,
                           typename V4<R>::type* __restrict__ vs)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    const int a = slot_atom[s];
    typename V4<R>::type o;
    o.x = 0; o.y = 0; o.z = 0; o.w = 0;
    if (a >= 0) {
        o.x = (R)v[3 * a];
        o.y = (R)v[3 * a + 1];
        o.z = (R)v[3 * a + 2];
    }
    vs[s] = o;
}

// Arguments of the adjoint pair kernel: the forward kernel's constants of the
// precision, and what the derivatives need.
template <typename R> struct AdjConst;
template <> struct AdjConst<float> { using K = PairConstF; using Shifts = ShiftTable; };
template <> struct AdjConst<double> { using K = PairConstD; using Shifts = ShiftTableD; };

template <typename R>
struct AdjArgs {
    int nlist;
    const ILRange* ilist;
    const PairEntry* plist;
    const typename V4<R>::type *xq, *vs;
    const int* stype;
    const float4* centerf;
    const double4* center;
    const int* nbidx;
    int ntp;
    int hot[2];         // the system's two most frequent atom types
    R gE, kc;
    typename AdjConst<R>::K K;
    typename AdjConst<R>::Shifts shifts;
    EwaldPoly poly;     // FP64
    int nlj;
    unsigned long long* dq_slot;
    double* dab;
    int n_ljpair;
    unsigned* st;
};

// erfc(alpha r)/r and its force factor times k, as the forward kernels.
template <bool POLY>
__device__ __forceinline__ void adj_ewald(const AdjArgs<float>& A, const PairConstF& K, float r2, float r, float rinv,
                                          float rinv2, float& e0, float& g0)
{
    const float ex = ex2_approx(K.kex * r2);
    e0 = A.kc * erfc_as(rcp_ftz(fmaf(K.pa, r, 1.0f)), ex) * rinv;
    g0 = fmaf(A.kc * K.two_a_spi, ex, e0) * rinv2;
}
template <bool POLY>
__device__ __forceinline__ void adj_ewald(const AdjArgs<double>& A, const PairConstD& K, double r2, double r,
                                          double rinv, double rinv2, double& e0, double& g0)
{
    double e, f;
    ewald_f64<POLY, true>(A.poly, K, r2, r, rinv, rinv2, e, f);
    e0 = A.kc * e;
    g0 = A.kc * f;
}

__device__ __forceinline__ float adj_rsqrt(float x) { return rsqrt_ftz(x); }
__device__ __forceinline__ double adj_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float adj_sat(float x) { return __saturatef(x); }
__device__ __forceinline__ double adj_sat(double x) { return fmax(0.0, x); }
__device__ __forceinline__ float adj_rc(const PairConstF& K) { return K.rcf; }
__device__ __forceinline__ double adj_rc(const PairConstD& K) { return K.rc; }

// Adjoint pair kernel: the forward kernel's warp layout (warp per i cluster,
// lane = (j slot, i atom), the j accumulator rotating one lane per step, j
// clusters staged twice so a step's atom sits at a compile-time offset) and its
// branch-free arithmetic; a slot outside the list or the cutoff adds zero.
//
// dL/dA and dL/dB go to the LJ entry of the pair's types.  A lane's i atom is
// fixed, so its pairs with the two most frequent atom types (of a solvated
// system, nearly all pairs) have two entries known before the loop: their sums
// stay in registers, and only pairs with other types add to the block's sums
// in shared memory at once.  (Runs of one entry, flushed when it changes, change
// at almost every pair, 32 lanes adding to a handful of shared words.)
//
// What bounds it: issue in FP32, the double-precision pipe in FP64.  28,000
// atoms: FP32 250 -> 93 us, FP64 521 -> 205 us (with the Ewald polynomials).
//
// Shared memory: staged positions, v and types of the warps' j clusters, then
// 2 * nlj partial sums (dA | dB) when nlj > 0; nlj == 0 sends every LJ term
// straight to global memory.
template <typename R, bool SWITCH, bool POLY>
__global__ void __launch_bounds__(NB_THREADS, sizeof(R) == 4 ? 3 : 2) k_adj_pairs(const __grid_constant__ AdjArgs<R> A)
{
    using V4t = typename V4<R>::type;
    extern __shared__ __align__(16) unsigned char adj_smem[];
    V4t* sx = reinterpret_cast<V4t*>(adj_smem);                          // [NB_WARPS][4][16]
    V4t* sv = sx + NB_WARPS * 4 * 2 * CLUSTER;                           // [NB_WARPS][4][16]
    int* stj = reinterpret_cast<int*>(sv + NB_WARPS * 4 * 2 * CLUSTER);  // [NB_WARPS][4][16]
    R* part = reinterpret_cast<R*>(stj + NB_WARPS * 4 * 2 * CLUSTER);    // [2 * nlj]
    constexpr int NS = sizeof(R) == 4 ? 6 : 3;
    __shared__ R sh[27][NS];
    for (int k = threadIdx.x; k < 27 * NS; k += blockDim.x) sh[k / NS][k % NS] = A.shifts.v[k / NS][k % NS];
    const int nlj = A.nlj;
    for (int k = threadIdx.x; k < 2 * nlj; k += blockDim.x) part[k] = (R)0;
    __syncthreads();
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * NB_WARPS + wib;
    const int jslot = lane >> 3, ii = lane & 7;
    const unsigned FULL = 0xffffffffu;
    const typename AdjConst<R>::K K = A.K;
    const R gE = A.gE;
    auto add_lj = [&](int k, R a, R b) {
        if (nlj > 0) {
            atomicAdd(part + k, a);
            atomicAdd(part + nlj + k, b);
        } else {
            atomicAdd(A.dab + k, (double)a);
            atomicAdd(A.dab + A.n_ljpair + k, (double)b);
        }
    };
    if (w < A.nlist) {
        const ILRange L = A.ilist[w];
        const int I = L.i;
        const V4t xi = A.xq[I * CLUSTER + ii];
        const V4t vi = A.vs[I * CLUSTER + ii];
        const int trow = A.stype[I * CLUSTER + ii] * A.ntp;
        const int k0 = A.nbidx[trow + A.hot[0]], kh = A.nbidx[trow + A.hot[1]], k1 = kh != k0 ? kh : -1;
        const int rot_src = (lane & ~7) | ((ii + 1) & 7);
        R dqi = 0, a0 = 0, b0 = 0, a1 = 0, b1 = 0;
        V4t* wsx = sx + (wib * 4 + jslot) * 2 * CLUSTER + ii;
        V4t* wsv = sv + (wib * 4 + jslot) * 2 * CLUSTER + ii;
        int* wst = stj + (wib * 4 + jslot) * 2 * CLUSTER + ii;
        for (int b = 0; b < L.count; b += 4) {
            const int e = b + jslot;
            PairEntry pe;
            if (e < L.count) {
                pe = A.plist[L.start + e];
            } else {
                pe.j = I; pe.shift = 13; pe.mask = 0ull;
            }
            const int J = pe.j;
            const V4t xjj = A.xq[J * CLUSTER + ii], vjj = A.vs[J * CLUSTER + ii];
            const int tjj = A.stype[J * CLUSTER + ii];
            wsx[0] = xjj; wsx[CLUSTER] = xjj;
            wsv[0] = vjj; wsv[CLUSTER] = vjj;
            wst[0] = tjj; wst[CLUSTER] = tjj;
            const R* s3 = sh[pe.shift];
            R xix, xiy, xiz;
            if constexpr (sizeof(R) == 4) {
                const float4 cI = A.centerf[I], cJ = A.centerf[J];
                xix = xi.x + (((cI.x - cJ.x) - s3[0]) - s3[3]);
                xiy = xi.y + (((cI.y - cJ.y) - s3[1]) - s3[4]);
                xiz = xi.z + (((cI.z - cJ.z) - s3[2]) - s3[5]);
            } else {
                const double4 cI = A.center[I], cJ = A.center[J];
                xix = xi.x + ((cI.x - cJ.x) - s3[0]);
                xiy = xi.y + ((cI.y - cJ.y) - s3[1]);
                xiz = xi.z + ((cI.z - cJ.z) - s3[2]);
            }
            const unsigned rowm = (unsigned)(pe.mask >> (ii * 8)) & 0xffu;
            const unsigned rot = ((rowm >> ii) | (rowm << (8 - ii))) & 0xffu;
            __syncwarp();
            R dqj = 0;
#pragma unroll
            for (int t = 0; t < CLUSTER; ++t) {
                const V4t xj = wsx[t], vj = wsv[t];
                const R dx = xix - xj.x, dy = xiy - xj.y, dz = xiz - xj.z;
                const R r2r = fma(dx, dx, fma(dy, dy, dz * dz));
                const bool on = ((rot >> t) & 1u) && r2r <= K.rc2;
                const R r2 = on ? r2r : (R)K.rc2;
                const R wv = fma(vi.x - vj.x, dx, fma(vi.y - vj.y, dy, (vi.z - vj.z) * dz));
                const R rinv = adj_rsqrt(r2), r = r2 * rinv, rinv2 = rinv * rinv;
                R e0, g0;
                adj_ewald<POLY>(A, K, r2, r, rinv, rinv2, e0, g0);
                R psi = fma(gE, e0, g0 * wv);
                psi = on ? psi : (R)0;
                dqi = fma(xj.w, psi, dqi);
                dqj = fma(xi.w, psi, dqj);
                // Lennard-Jones: E = A eA + B eB, g = A gA + B gB
                const R rinv6 = rinv2 * rinv2 * rinv2;
                R da, db;
                if (SWITCH) {
                    const R x = adj_sat(fma(r, K.inv_sw, -K.rsw_inv)), x2 = x * x;
                    const R S = fma(x2 * x, fma(x, fma(x, (R)-6, (R)15), (R)-10), (R)1);
                    const R dSr = x2 * fma(x, fma(x, K.d30, K.d60), K.d30) * rinv;   // dS/dr / r
                    const R base = fma(gE, S, -wv * dSr), sw = wv * rinv2 * S;
                    da = rinv6 * rinv6 * fma((R)12, sw, base);
                    db = -rinv6 * fma((R)6, sw, base);
                } else {
                    // force-shifted: U - U(rc) + (r - rc) g(rc) rc, linear in A and B
                    const R rc = adj_rc(K);
                    const R gcA = (R)12 * K.uc12 / K.rc2 * rc, gcB = (R)-6 * K.uc6 / K.rc2 * rc;
                    const R eA = rinv6 * rinv6 - K.uc12 + (r - rc) * gcA, eB = -rinv6 + K.uc6 + (r - rc) * gcB;
                    const R gA = (R)12 * rinv6 * rinv6 * rinv2 - gcA * rinv, gB = (R)-6 * rinv6 * rinv2 - gcB * rinv;
                    da = fma(gE, eA, gA * wv);
                    db = fma(gE, eB, gB * wv);
                }
                const int k = on ? A.nbidx[trow + wst[t]] : -1;
                const bool h0 = k >= 0 && k == k0, h1 = k >= 0 && k == k1;
                a0 += h0 ? da : (R)0;
                b0 += h0 ? db : (R)0;
                a1 += h1 ? da : (R)0;
                b1 += h1 ? db : (R)0;
                if (k >= 0 && !h0 && !h1) add_lj(k, da, db);
                dqj = __shfl_sync(FULL, dqj, rot_src);
            }
            if (e < L.count && dqj != (R)0) fx_add(A.dq_slot + J * CLUSTER + ii, (double)dqj, FORCE_SCALE, A.st);
            __syncwarp();
        }
        dqi += __shfl_xor_sync(FULL, dqi, 8);
        dqi += __shfl_xor_sync(FULL, dqi, 16);
        if (jslot == 0 && dqi != (R)0) fx_add(A.dq_slot + I * CLUSTER + ii, (double)dqi, FORCE_SCALE, A.st);
        if (k0 >= 0) add_lj(k0, a0, b0);
        if (k1 >= 0) add_lj(k1, a1, b1);
    }
    if (nlj > 0) {
        __syncthreads();
        for (int k = threadIdx.x; k < 2 * nlj; k += blockDim.x) {
            const R v = part[k];
            if (v != (R)0) atomicAdd(A.dab + (k < nlj ? k : A.n_ljpair + k - nlj), (double)v);
        }
    }
}

// Excluded pairs (-k q q erf(alpha r)/r) and 1-4 Coulomb pairs (k q q/(scee r)),
// FP64, minimum image, atom order.
__global__ void k_adj_pairs_fp64(int nex, const int* __restrict__ excl, int n14, const int* __restrict__ p14,
                                 const double2* __restrict__ scale14, const double* __restrict__ xyz,
                                 const double* __restrict__ q, const double* __restrict__ v, NBParams P, double gE,
                                 unsigned long long* __restrict__ dq, unsigned* st)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nex + n14) return;
    const bool ex = k < nex;
    const int a = ex ? excl[2 * k] : p14[2 * (k - nex)], b = ex ? excl[2 * k + 1] : p14[2 * (k - nex) + 1];
    double d[3];
    for (int c = 0; c < 3; ++c) d[c] = min_image(xyz[3 * a + c] - xyz[3 * b + c], P.box[c]);
    const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2], r = sqrt(r2);
    double e0, g0;
    if (ex) {
        const double ar = P.alpha * r;
        e0 = -P.kc * erf(ar) / r;
        g0 = (e0 + P.kc * (2.0 * P.alpha / 1.7724538509055160273) * exp(-ar * ar)) / r2;
    } else {
        e0 = P.kc / (scale14[k - nex].x * r);
        g0 = e0 / r2;
    }
    const double w = (v[3 * a] - v[3 * b]) * d[0] + (v[3 * a + 1] - v[3 * b + 1]) * d[1] +
                     (v[3 * a + 2] - v[3 * b + 2]) * d[2];
    const double psi = gE * e0 + g0 * w;
    fx_add(dq + a, q[b] * psi, FORCE_SCALE, st);
    fx_add(dq + b, q[a] * psi, FORCE_SCALE, st);
}

// Self energy and net-charge term, and the final sum (atom order, unscaled).
__global__ void k_adj_finish(int N, const double* __restrict__ q, const int* __restrict__ atom_slot,
                             const unsigned long long* __restrict__ dq_atom,
                             const unsigned long long* __restrict__ dq_slot, double self_coef, double net_coef,
                             double scale, double* __restrict__ out)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= N) return;
    const long long f = (long long)dq_atom[a] + (long long)dq_slot[atom_slot[a]];
    out[a] = ((double)f * FORCE_ISCALE + self_coef * q[a] + net_coef) * scale;
}

__global__ void k_scale(int n, double* __restrict__ x, double s)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] *= s;
}

static void adj_consts(const Ctx& c, AdjArgs<float>& A)
{
    const PairF32Args F = make_pair_f32_args(c, nullptr);
    A.K = F.K;
    A.shifts = F.shifts;
    A.xq = c.xq_f.p;
}
static void adj_consts(const Ctx& c, AdjArgs<double>& A)
{
    const PairF64Args F = make_pair_f64_args(c, nullptr);
    A.K = F.K;
    A.shifts = F.shifts;
    A.poly = F.poly;
    A.xq = c.xq_d.p;
}

template <typename R>
static void launch_adj_pairs(Ctx& c, const NBParams& P, double gE, const AdjBufs& M)
{
    AdjArgs<R> A{};
    adj_consts(c, A);
    A.vs = reinterpret_cast<const typename V4<R>::type*>(M.vs);
    const bool pruned = c.p.prune_every != 0;   // backward() has just pruned whole entries
    A.nlist = c.n_clusters;
    A.ilist = pruned ? c.ilist_in.p : c.ilist.p;
    A.plist = pruned ? c.plist_in.p : c.plist.p;
    A.stype = c.slot_type.p;
    A.centerf = c.centerf.p;
    A.center = c.center.p;
    A.nbidx = c.nbidx.p;
    A.ntp = c.ntp;
    A.hot[0] = c.hot_type[0];
    A.hot[1] = c.hot_type[1];
    A.gE = (R)gE;
    A.kc = (R)P.kc;
    A.dq_slot = M.dq_slot;
    A.dab = M.dab;
    A.n_ljpair = c.n_ljpair;
    A.st = c.status.p;
    const size_t stage = (size_t)NB_WARPS * 4 * 2 * CLUSTER * (2 * sizeof(typename V4<R>::type) + sizeof(int));
    A.nlj = c.n_ljpair;
    size_t smem = stage + 2 * (size_t)A.nlj * sizeof(R);
    if (smem > 96 * 1024) {   // too many LJ entries for per-block partials: global atomics
        A.nlj = 0;
        smem = stage;
    }
    auto go = [&](auto kern) {
        MDF_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid_blocks(c.n_clusters, NB_WARPS), NB_THREADS, smem, c.stream>>>(A);
    };
    if (P.use_switch) {
        if (A.poly.on) go(k_adj_pairs<R, true, true>);
        else go(k_adj_pairs<R, true, false>);
    } else {
        if (A.poly.on) go(k_adj_pairs<R, false, true>);
        else go(k_adj_pairs<R, false, false>);
    }
    MDF_CUDA_TRY(cudaGetLastError());
}

// The call's buffers; slots by the list's capacity, so that a rebuilt list
// rarely asks for more.
static AdjBufs adj_bufs(Ctx& c)
{
    const bool mixed = c.p.precision == MDF_PREC_MIXED;
    const size_t N = c.N, slots = c.slot_atom.n, ntot = (size_t)c.K[0] * c.K[1] * c.K[2];
    const size_t nc = (size_t)c.K[0] * c.K[1] * (c.K[2] / 2 + 1);
    const size_t bytes[8] = {sizeof(double) * 3 * N,
                             (mixed ? sizeof(float4) : sizeof(double4)) * slots,
                             sizeof(unsigned long long) * slots,
                             sizeof(unsigned long long) * N,
                             sizeof(double) * 2 * (size_t)c.n_ljpair,
                             sizeof(double) * N,
                             sizeof(unsigned long long) * ntot,
                             (mixed ? sizeof(float2) : sizeof(double2)) * nc};
    size_t off[9] = {0};
    for (int i = 0; i < 8; ++i) off[i + 1] = off[i] + (bytes[i] + 255) / 256 * 256;
    c.adj_mem.alloc(off[8]);
    unsigned char* p = c.adj_mem.p;
    return AdjBufs{reinterpret_cast<double*>(p + off[0]),
                   p + off[1],
                   reinterpret_cast<unsigned long long*>(p + off[2]),
                   reinterpret_cast<unsigned long long*>(p + off[3]),
                   reinterpret_cast<double*>(p + off[4]),
                   reinterpret_cast<double*>(p + off[5]),
                   reinterpret_cast<unsigned long long*>(p + off[6]),
                   p + off[7]};
}

void backward(Ctx& c, const double* dL_dF, double dL_dE, double* dL_dq, double* dL_dA, double* dL_dB)
{
    if (c.p.semantics != MDF_SEM_PHYSICAL)
        throw ApiError(MDF_ERR_UNSUPPORTED, "mdf_backward needs PHYSICAL semantics (REFERENCE forces are not "
                                            "the gradient of its energy)");
    if (!c.have_positions) throw ApiError(MDF_ERR_STATE, "positions not set");
    if (!c.have_list) build_pairlist(c);
    cudaStream_t s = c.stream;
    const bool mixed = c.p.precision == MDF_PREC_MIXED;
    // normalise: scale = max(|gE|, max |v|)
    double scale = std::fabs(dL_dE);
    if (dL_dF)
        for (long long i = 0; i < 3LL * c.N; ++i) scale = std::max(scale, std::fabs(dL_dF[i]));
    const int nlj = c.n_ljpair;
    if (scale == 0.0 || !std::isfinite(scale)) {
        if (!std::isfinite(scale)) throw ApiError(MDF_ERR_NONFINITE, "non-finite dL/dF or dL/dE");
        if (dL_dq) std::fill(dL_dq, dL_dq + c.N, 0.0);
        if (dL_dA) std::fill(dL_dA, dL_dA + nlj, 0.0);
        if (dL_dB) std::fill(dL_dB, dL_dB + nlj, 0.0);
        return;
    }
    std::vector<double> vn(3 * (size_t)c.N, 0.0);
    if (dL_dF)
        for (long long i = 0; i < 3LL * c.N; ++i) vn[i] = dL_dF[i] / scale;
    const double gE = dL_dE / scale;
    const AdjBufs M = adj_bufs(c);
    MDF_CUDA_TRY(cudaMemcpyAsync(M.v, vn.data(), sizeof(double) * vn.size(), cudaMemcpyHostToDevice, s));
    MDF_CUDA_TRY(cudaMemsetAsync(M.dq_slot, 0, sizeof(unsigned long long) * c.n_slots, s));
    MDF_CUDA_TRY(cudaMemsetAsync(M.dq_atom, 0, sizeof(unsigned long long) * c.N, s));
    if (nlj > 0) MDF_CUDA_TRY(cudaMemsetAsync(M.dab, 0, sizeof(double) * 2 * nlj, s));
    MDF_CUDA_TRY(cudaMemsetAsync(c.status.p, 0, sizeof(unsigned), s));
    const int th = 256;
    // current cluster frame and pruned list, as a forward evaluation builds them
    pack_positions(c);
    if (c.p.prune_every != 0) {
        prune_pairlist(c, true);   // whole entries: the adjoint kernel walks 8 x 8 cluster pairs
        c.since_prune = 1;
        if (half_layout(c)) c.pruned_valid = false;   // the next forward prunes its half lists again
    }
    if (mixed)
        k_adj_pack<float><<<grid_blocks(c.n_slots, th), th, 0, s>>>(c.n_slots, c.slot_atom.p, M.v,
                                                                     reinterpret_cast<float4*>(M.vs));
    else
        k_adj_pack<double><<<grid_blocks(c.n_slots, th), th, 0, s>>>(c.n_slots, c.slot_atom.p, M.v,
                                                                      reinterpret_cast<double4*>(M.vs));
    const NBParams P = make_params(c);
    // the reciprocal-space part runs on the side stream, concurrently with
    // the pair adjoint (both only add into the fixed-point dq accumulators)
    MDF_CUDA_TRY(cudaEventRecord(c.ev_fork, s));
    MDF_CUDA_TRY(cudaStreamWaitEvent(c.side, c.ev_fork, 0));
    c.stream = c.side;
    try {
        pme_adjoint(c, gE, M);
    } catch (...) {
        c.stream = s;
        throw;
    }
    c.stream = s;
    MDF_CUDA_TRY(cudaEventRecord(c.ev_join, c.side));
    if (mixed) launch_adj_pairs<float>(c, P, gE, M);
    else launch_adj_pairs<double>(c, P, gE, M);
    if (c.n_excl + c.n_14 > 0)
        k_adj_pairs_fp64<<<grid_blocks(c.n_excl + c.n_14, th), th, 0, s>>>(
            c.n_excl, c.excl_pairs.p, c.n_14, c.pairs14.p, c.p14_scale.p, c.xyz.p, c.q.p, M.v, P, gE,
            M.dq_atom, c.status.p);
    MDF_CUDA_TRY(cudaStreamWaitEvent(s, c.ev_join, 0));
    // d/dq_a of gE (E_self + E_net): -2 k alpha/sqrt(pi) q_a and -k pi Q / (V alpha^2)
    const double V = c.box[0] * c.box[1] * c.box[2];
    const double self_coef = gE * (-2.0 * c.p.coulomb_const * c.alpha / std::sqrt(M_PI));
    const double net_coef = gE * (-c.p.coulomb_const * M_PI * c.q_total / (V * c.alpha * c.alpha));
    k_adj_finish<<<grid_blocks(c.N, th), th, 0, s>>>(c.N, c.q.p, c.atom_slot.p, M.dq_atom, M.dq_slot, self_coef,
                                                     net_coef, scale, M.dq);
    if (nlj > 0) k_scale<<<grid_blocks(2 * nlj, th), th, 0, s>>>(2 * nlj, M.dab, scale);
    MDF_CUDA_TRY(cudaGetLastError());
    c.launches += 6;
    unsigned st = 0;
    MDF_CUDA_TRY(cudaMemcpyAsync(&st, c.status.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    if (dL_dq) MDF_CUDA_TRY(cudaMemcpyAsync(dL_dq, M.dq, sizeof(double) * c.N, cudaMemcpyDeviceToHost, s));
    if (dL_dA && nlj > 0)
        MDF_CUDA_TRY(cudaMemcpyAsync(dL_dA, M.dab, sizeof(double) * nlj, cudaMemcpyDeviceToHost, s));
    if (dL_dB && nlj > 0)
        MDF_CUDA_TRY(cudaMemcpyAsync(dL_dB, M.dab + nlj, sizeof(double) * nlj, cudaMemcpyDeviceToHost, s));
    // the status word belongs to the forward's scalar block: leave it clear
    MDF_CUDA_TRY(cudaMemsetAsync(c.status.p, 0, sizeof(unsigned), s));
    MDF_CUDA_TRY(cudaStreamSynchronize(s));
    if (st & ST_NONFINITE) throw ApiError(MDF_ERR_NONFINITE, "non-finite value in the adjoint");
    if (st & ST_OVERFLOW) throw ApiError(MDF_ERR_OVERFLOW, "fixed-point accumulator range exceeded in the adjoint");
}

}  // namespace mdf
