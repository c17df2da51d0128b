// Cluster sort and cluster-pair list (replaces the reference's linked-list
// cell pairlist, src/System/NonBondedUtils.cpp:185-282).
//
// Atoms are binned into x-y columns whose cross-section holds about one
// cluster-height of atoms, sorted by z inside each column, and cut into
// clusters of 8; columns are numbered x-major (y fastest), so consecutive
// clusters sweep a band of x.  Every i cluster then gets the list of j clusters (j >= i,
// half list) whose bounding boxes, in some periodic image, come within the
// list cutoff (cutoff + skin).  Each entry carries a 64-bit mask of the atom
// pairs that interact: padding slots, the lower triangle of the self pair and
// excluded pairs are cleared.
#include <algorithm>
#include <cmath>

#include "bands.hpp"
#include "kargs.cuh"
#include "mdf_device.cuh"
#include "mdf_internal.cuh"

namespace mdf {

int grid_blocks(long long n, int threads)
{
    long long b = (n + threads - 1) / threads;
    return (int)std::max(1LL, b);
}

// ------------------------------------------------------------------ scan
// Column table in one block: exclusive scans of the atom counts (col_start)
// and of the cluster counts (col_cstart, ceil(count / 8) per column), and the
// cluster total at col_cstart[ncols].  A column above COL_MAX atoms (the
// in-block sort's limit) sets ST_CAPACITY_COLUMN.  ncols is at most a few
// thousand, so each thread takes a contiguous chunk.
constexpr int COL_MAX = 2048;   // atoms per column handled by the in-block sort

__global__ void __launch_bounds__(1024) k_column_table(int ncols, const int* __restrict__ cnt,
                                                       int* __restrict__ col_start, int* __restrict__ col_cstart,
                                                       unsigned* st)
{
    __shared__ int part_a[1024], part_c[1024];
    const int tid = threadIdx.x, per = (ncols + blockDim.x - 1) / blockDim.x;
    const int b0 = min(ncols, tid * per), b1 = min(ncols, b0 + per);
    int sa = 0, sc = 0;
    bool over = false;
    for (int i = b0; i < b1; ++i) {
        const int n = cnt[i];
        sa += n;
        sc += (n + CLUSTER - 1) / CLUSTER;
        over = over || n > COL_MAX;
    }
    if (over) status_set(st, ST_CAPACITY_COLUMN);
    part_a[tid] = sa;
    part_c[tid] = sc;
    __syncthreads();
    for (int o = 1; o < blockDim.x; o <<= 1) {   // Hillis-Steele inclusive scan of the partials
        const int va = tid >= o ? part_a[tid - o] : 0, vc = tid >= o ? part_c[tid - o] : 0;
        __syncthreads();
        part_a[tid] += va;
        part_c[tid] += vc;
        __syncthreads();
    }
    int ra = tid ? part_a[tid - 1] : 0, rc = tid ? part_c[tid - 1] : 0;
    for (int i = b0; i < b1; ++i) {
        const int n = cnt[i];
        col_start[i] = ra;
        col_cstart[i] = rc;
        ra += n;
        rc += (n + CLUSTER - 1) / CLUSTER;
    }
    if (tid == blockDim.x - 1) {
        col_start[ncols] = part_a[tid];
        col_cstart[ncols] = part_c[tid];
    }
}

// ------------------------------------------------------------- binning
// Each atom's column, and its place among the column's atoms in the order of
// arrival (the sort that follows makes the order a fixed one).  Neighbouring
// atoms mostly share a column: one addition per column and warp.
__global__ void k_assign_columns(int N, const double* __restrict__ xyz, double Lx, double Ly, int ncx, int ncy,
                                 int2* __restrict__ atom_col, int* __restrict__ col_count, unsigned* st)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned live = __ballot_sync(0xffffffffu, i < N);
    if (i >= N) return;
    double x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    if (!isfinite(x) || !isfinite(y) || !isfinite(z)) {
        status_set(st, ST_NONFINITE);
        x = y = 0.0;
    }
    x = wrap_coord(x, Lx);
    y = wrap_coord(y, Ly);
    int cx = (int)(x * ncx / Lx), cy = (int)(y * ncy / Ly);
    cx = min(max(cx, 0), ncx - 1);
    cy = min(max(cy, 0), ncy - 1);
    // x-major: consecutive columns run along y, so a contiguous range of
    // clusters is a band of x (a split evaluation's share of space)
    int col = cy + ncy * cx;
    const unsigned same = __match_any_sync(live, col);
    const int lane = threadIdx.x & 31, lead = __ffs(same) - 1;
    int first = 0;
    if (lane == lead) first = atomicAdd(&col_count[col], __popc(same));
    first = __shfl_sync(same, first, lead);
    atom_col[i] = make_int2(col, first + __popc(same & ((1u << lane) - 1u)));
}

__global__ void k_bucket(int N, const int2* __restrict__ atom_col, const int* __restrict__ col_start,
                         int* __restrict__ col_atoms)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int2 c = atom_col[i];
    col_atoms[col_start[c.x] + c.y] = i;
}

// One block per column: bitonic sort of (z, atom) keys, then cut into clusters
// of 8.  A column holds ~200 atoms at liquid density, so 256 threads cover the
// exchanges of a step, and its barriers wait for 8 warps instead of 32
// (100k atoms 21.7 -> 12.5 us).
constexpr int SORT_THREADS = 256;

__global__ void __launch_bounds__(SORT_THREADS) k_sort_columns(const double* __restrict__ xyz, double Lz,
                                                       const int* __restrict__ col_count,
                                                       const int* __restrict__ col_start,
                                                       const int* __restrict__ col_cstart,
                                                       const int* __restrict__ col_atoms,
                                                       int* __restrict__ slot_atom, int* __restrict__ atom_slot,
                                                       int* __restrict__ cluster_col, unsigned* st)
{
    __shared__ unsigned long long key[COL_MAX];
    int col = blockIdx.x, tid = threadIdx.x;
    int n = col_count[col];
    int s0 = col_start[col];
    if (n > COL_MAX) {
        // The build restarts with thinner columns; until then this column's
        // clusters are left empty and its atoms point at slot 0, so the
        // kernels queued after this one only touch valid memory.
        if (tid == 0) status_set(st, ST_CAPACITY_COLUMN);
        const int c0 = col_cstart[col], ncl = (n + CLUSTER - 1) / CLUSTER;
        for (int k = tid; k < ncl * CLUSTER; k += blockDim.x) {
            slot_atom[c0 * CLUSTER + k] = -1;
            if ((k % CLUSTER) == 0) cluster_col[c0 + k / CLUSTER] = col;
        }
        for (int k = tid; k < n; k += blockDim.x) atom_slot[col_atoms[s0 + k]] = 0;
        return;
    }
    // pad to the next power of two >= n (at least 2)
    int m = 2;
    while (m < n) m <<= 1;
    for (int k = tid; k < m; k += blockDim.x) {
        unsigned long long kk = ~0ull;
        if (k < n) {
            int a = col_atoms[s0 + k];
            double zw = wrap_coord(xyz[3 * a + 2], Lz);
            float zf = (float)zw;
            if (!(zf >= 0.0f)) zf = 0.0f;
            kk = ((unsigned long long)__float_as_uint(zf) << 32) | (unsigned)a;
        }
        key[k] = kk;
    }
    for (int size = 2; size <= m; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int t = tid; t < (m >> 1); t += blockDim.x) {
                int i = 2 * t - (t & (stride - 1));
                int j = i + stride;
                bool asc = (i & size) == 0;
                unsigned long long a = key[i], b = key[j];
                if ((a > b) == asc) {
                    key[i] = b;
                    key[j] = a;
                }
            }
        }
    }
    __syncthreads();
    int c0 = col_cstart[col];
    int ncl = (n + CLUSTER - 1) / CLUSTER;
    for (int k = tid; k < ncl * CLUSTER; k += blockDim.x) {
        int cl = c0 + k / CLUSTER;
        int slot = cl * CLUSTER + (k % CLUSTER);
        if (k < n) {
            int a = (int)(key[k] & 0xffffffffu);
            slot_atom[slot] = a;
            atom_slot[a] = slot;
        } else {
            slot_atom[slot] = -1;
        }
        if ((k % CLUSTER) == 0) cluster_col[cl] = col;
    }
}

// Cluster bounding boxes (wrapped coordinates; bb_lo.w = number of real atoms),
// centres (center.w the same) and the slots' types.  Eight lanes per cluster,
// launched over the slot capacity; the clusters the column table made (*d_ncl)
// are the ones with work.  blockDim.x must be a multiple of 32.
__global__ void k_cluster_geom(const int* __restrict__ d_ncl, const double* __restrict__ xyz, double Lx, double Ly,
                               double Lz, double quantum, const int* __restrict__ slot_atom,
                               const int* __restrict__ type, int pad_type, double4* __restrict__ center,
                               float4* __restrict__ centerf, float4* __restrict__ bb_lo, float4* __restrict__ bb_hi,
                               int* __restrict__ slot_type)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x, c = s / CLUSTER;
    const bool inside = c < *d_ncl;
    const int a = inside ? slot_atom[s] : -1;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    int nv = 0;
    if (a >= 0) {
        nv = 1;
        lo[0] = hi[0] = wrap_coord(xyz[3 * a], Lx);
        lo[1] = hi[1] = wrap_coord(xyz[3 * a + 1], Ly);
        lo[2] = hi[2] = wrap_coord(xyz[3 * a + 2], Lz);
    }
#pragma unroll
    for (int o = 1; o < CLUSTER; o <<= 1) {
        nv += __shfl_xor_sync(0xffffffffu, nv, o);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    }
    if (!inside) return;
    slot_type[s] = a < 0 ? pad_type : type[a];
    if (s % CLUSTER) return;
    if (nv == 0) {
        for (int d = 0; d < 3; ++d) lo[d] = hi[d] = 0.0;
    }
    // centres on a 2^-k grid fine enough that they are exact in FP32, so the
    // FP32 pair kernel forms centre differences without rounding
    double cc[3];
    for (int d = 0; d < 3; ++d) cc[d] = rint(0.5 * (lo[d] + hi[d]) / quantum) * quantum;
    center[c] = make_double4(cc[0], cc[1], cc[2], (double)nv);
    centerf[c] = make_float4((float)cc[0], (float)cc[1], (float)cc[2], (float)nv);
    bb_lo[c] = make_float4(__double2float_rd(lo[0]), __double2float_rd(lo[1]), __double2float_rd(lo[2]), (float)nv);
    bb_hi[c] = make_float4(__double2float_ru(hi[0]), __double2float_ru(hi[1]), __double2float_ru(hi[2]), 0.f);
}

struct BoxF {
    float x, y, z, hx, hy, hz;
    bool fine;   // half extents to 1/64 A
};

// Box of a cluster in absolute coordinates: centre, and half extents in units
// of 2^(6s-6) A, rounded up, as 3 x 10 bits with s in the top two (up to 4.1e6 A,
// a box of 0.8 mm).
__device__ __forceinline__ float4 box_encode(const float lo[3], const float hi[3], const double4& c, float pad)
{
    float h[3], m = 0.f;
    for (int k = 0; k < 3; ++k) {
        h[k] = fmaxf(0.f, 0.5f * (hi[k] - lo[k])) + pad;   // + rounding of the centre
        m = fmaxf(m, h[k]);
    }
    unsigned s = 0;
    while (s < 3 && m > 1020.f * __uint_as_float((121u + 6u * s) << 23)) ++s;
    const float per = __uint_as_float((133u - 6u * s) << 23);   // 2^(6-6s)
    unsigned u = s << 30;
    for (int k = 0; k < 3; ++k) u |= min(1023u, (unsigned)ceilf(h[k] * per)) << (10 * k);
    const bool real = lo[0] <= hi[0];
    return make_float4((float)c.x + (real ? 0.5f * (lo[0] + hi[0]) : 0.f),
                       (float)c.y + (real ? 0.5f * (lo[1] + hi[1]) : 0.f),
                       (float)c.z + (real ? 0.5f * (lo[2] + hi[2]) : 0.f), __uint_as_float(u));
}

__device__ __forceinline__ BoxF box_decode(const float4& b)
{
    const unsigned u = __float_as_uint(b.w);
    const float unit = __uint_as_float((121u + 6u * (u >> 30)) << 23);
    return BoxF{b.x, b.y, b.z, (float)(u & 1023u) * unit, (float)((u >> 10) & 1023u) * unit,
                (float)((u >> 20) & 1023u) * unit, (u >> 30) == 0u};
}

// Per-evaluation packing: cluster-ordered offsets from the cluster centre
// (min image, so atoms crossing the box edge between rebuilds stay whole)
// plus charge, in the working precision.
// Also the cluster's current bounding box for the prune's box test
// (box_encode) and, in FP64, the FP32 copy of the offsets that the prune reads.
// blockDim.x must be a multiple of 32.
template <typename R>
__device__ __forceinline__ void pack_dev(const PackArgs<R>& A, int bx, int by)
{
    const int nslots = A.nslots;
    const double* __restrict__ xyz = A.xyz;
    const double* __restrict__ q = A.q;
    const int* __restrict__ slot_atom = A.slot_atom;
    const double4* __restrict__ center = A.center;
    const double Lx = A.L[0], Ly = A.L[1], Lz = A.L[2];
    typename V4<R>::type* __restrict__ xq = A.xq;
    unsigned* st = A.st;
    const int s = bx * blockDim.x + threadIdx.x;
    const bool inside = s < nslots;
    const int a = inside ? slot_atom[s] : -1;
    typename V4<R>::type v;
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    if (a < 0) {
        v.x = v.y = v.z = v.w = (R)0;
    } else {
        double4 c = center[s / CLUSTER];
        double d[3] = {min_image(xyz[3 * a] - c.x, Lx), min_image(xyz[3 * a + 1] - c.y, Ly),
                       min_image(xyz[3 * a + 2] - c.z, Lz)};
        if (!isfinite(d[0] + d[1] + d[2])) status_set(st, ST_NONFINITE);
        v.x = (R)d[0];
        v.y = (R)d[1];
        v.z = (R)d[2];
        v.w = (R)q[a];
        for (int k = 0; k < 3; ++k) {
            lo[k] = __double2float_rd(d[k]);
            hi[k] = __double2float_ru(d[k]);
        }
    }
    if (inside) xq[s] = v;
    if (sizeof(R) == 8 && inside) A.xf[s] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    if (A.snap) {
        // self-pruning: the largest squared displacement since the last prune
        float d2 = 0.f;
        if (a >= 0) {
            const typename V4<R>::type o = A.snap[s];
            const double ex = (double)v.x - (double)o.x, ey = (double)v.y - (double)o.y, ez = (double)v.z - (double)o.z;
            d2 = __double2float_ru(ex * ex + ey * ey + ez * ez);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d2 = fmaxf(d2, __shfl_xor_sync(0xffffffffu, d2, o));
        if ((threadIdx.x & 31) == 0 && d2 > 0.f) atomicMax(A.disp, __float_as_uint(d2));
    }
    // min/max over the 8 slots of the cluster (8 consecutive lanes)
#pragma unroll
    for (int o = 1; o < CLUSTER; o <<= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    if (inside && (s % CLUSTER) == 0) A.box[s / CLUSTER] = box_encode(lo, hi, center[s / CLUSTER], A.box_pad);
}

template <typename R>
__global__ void k_pack(PackArgs<R> A)
{
    pack_dev(A, blockIdx.x, 0);
}

template <typename R>
__global__ void k_pack_multi(const PackArgs<R>* __restrict__ As, const int2* __restrict__ bmap)
{
    const int2 m = bmap[blockIdx.x];
    pack_dev(As[m.x], m.y, 0);
}

// -------------------------------------------------------- pair search
struct SearchGeom {
    double L[3];
    double colw[3];
    int ncx, ncy;
    int Rx, Ry;
    float rlist2;
    float rlist;
};

// Interacting pairs of an entry before exclusions: real atoms of both clusters,
// jj > ii for the pair of a cluster with itself.
__device__ __forceinline__ unsigned long long entry_mask(int nvi, int nvj, bool self_pair)
{
    const unsigned long long row = (1ull << nvj) - 1ull;
    unsigned long long m = row * 0x0101010101010101ull;          // every i row (nvj <= 8)
    if (nvi < CLUSTER) m &= (1ull << (8 * nvi)) - 1ull;
    if (self_pair) m &= 0x0080c0e0f0f8fcfeull;                   // byte ii: bits above ii
    return m;
}

// Periodic image of atom b's cluster entry for an excluded pair (a in cluster
// I): the key (J << 5 | code) of the entry that holds the pair in I's list and
// the pair's bit, or false when the pair belongs to another list or to none.
__device__ __forceinline__ bool excluded_entry(int I, int la, int a, int b, const int* __restrict__ atom_slot,
                                               const double* __restrict__ xyz, const double4* __restrict__ center,
                                               const double L[3], unsigned& key, int& bit)
{
    const int sb = atom_slot[b], J = sb / CLUSTER, lb = sb % CLUSTER;
    if (J < I || (J == I && b < a)) return false;   // J's list holds it, or the pair comes up the other way round
    const double4 ca = center[I], cb = center[J];
    const double pca[3] = {ca.x, ca.y, ca.z}, pcb[3] = {cb.x, cb.y, cb.z};
    int code = 0, f = 1;
    for (int d = 0; d < 3; ++d) {
        // list-geometry positions: centre + min-image offset; J's atoms sit at
        // p + s L in I's frame: s = round((p_I - p_J) / L)
        const double pa = pca[d] + min_image(xyz[3 * a + d] - pca[d], L[d]);
        const double pb = pcb[d] + min_image(xyz[3 * b + d] - pcb[d], L[d]);
        const int s = (int)round((pa - pb) / L[d]);
        if (s < -1 || s > 1) return false;          // never listed
        code += f * (s + 1);
        f *= 3;
    }
    bit = la * 8 + lb;
    if (J == I) {
        if (code == 13) bit = min(la, lb) * 8 + max(la, lb);
        else if (code < 13) {
            bit = lb * 8 + la;
            code = 26 - code;
        }
    }
    key = ((unsigned)J << 5) | (unsigned)code;
    return true;
}

// Clusters beyond this extent (A) are pruned by the WIDE form.  Liquids stay at 5
// to 10 A, and a slab that straddles the box edge at the vacuum beside it: with
// a line at 64 A such a slab (100k atoms, 60 A of vacuum) took 64 us in the prune
// instead of 43, 102 instead of 44 in FP64.
constexpr float WIDE_EXTENT = 256.f;

constexpr int SEARCH_WARPS = 4;
constexpr int SEARCH_CAP = 512;   // entries a warp buffers (~125 per i cluster at liquid density, 10 + 2 A)

// One warp per i cluster (launched over the cluster capacity; clusters at or
// above *d_ncl return).  Lanes take the columns around the cluster and find
// each one's run of j clusters in the list's z range by bisection; the runs of
// 32 columns are then walked as one sequence, a lane per candidate, so boxes
// are read in order and every lane tests.  Columns before the own one hold only
// j < i and are skipped whole.  Entries collect in shared memory, the exclusion
// bits are cleared there - lanes look up the cluster's excluded partners and
// scan the entries together - and the range is claimed with one atomicAdd on
// *d_total and written coalesced.  The order inside a range is fixed (columns,
// images, j), so every evaluation sums the same terms in the same order; only
// the ranges' positions depend on the order the warps ran in.  A cluster with
// more than SEARCH_CAP entries generates them twice, the second time through
// the buffer in pieces.  Entries past `cap` are counted but not written
// (ST_CAPACITY_PAIRS: the host grows the list and searches again).
//
// A lane per column, counting and then writing, and a warp per excluded pair that
// searches its entry in global memory take 245 us where this takes 80 (100k
// atoms; 960k 2,235 and 730; a whole build 336 and 132 us, 2.56 and 0.86 ms).
__global__ void __launch_bounds__(32 * SEARCH_WARPS) k_pair_search(
    const int* __restrict__ d_ncl, const SearchGeom g, const int* __restrict__ cluster_col,
    const int* __restrict__ col_cstart, const float4* __restrict__ bb_lo, const float4* __restrict__ bb_hi,
    const double4* __restrict__ center, const int* __restrict__ slot_atom, const int* __restrict__ atom_slot,
    const double* __restrict__ xyz, const int* __restrict__ ex_off, const int* __restrict__ ex_nb,
    int* __restrict__ d_total, PairEntry* __restrict__ out, long long cap, ILRange* __restrict__ ilist, unsigned* st)
{
    __shared__ unsigned s_key[SEARCH_WARPS][SEARCH_CAP];
    __shared__ unsigned s_mask[SEARCH_WARPS][2 * SEARCH_CAP];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = blockIdx.x * SEARCH_WARPS + wib;
    if (I >= *d_ncl) return;
    unsigned* key = s_key[wib];
    unsigned* mask = s_mask[wib];
    const unsigned FULL = 0xffffffffu, below = (1u << lane) - 1u;
    const int col = cluster_col[I];
    const int cx = col / g.ncy, cy = col % g.ncy;
    const float4 lo = bb_lo[I], hi = bb_hi[I];
    if (lane == 0 && fmaxf(hi.x - lo.x, fmaxf(hi.y - lo.y, hi.z - lo.z)) > WIDE_EXTENT) d_total[1] = 1;
    const int nvi = (int)lo.w;
    const int nxc = 2 * g.Rx + 1, ncand = nxc * (2 * g.Ry + 1);
    const float Lx = (float)g.L[0], Ly = (float)g.L[1], Lz = (float)g.L[2];

    // The candidates of the list in their order; emit(mask of lanes with an entry, this lane's key).
    auto generate = [&](auto&& emit) {
        for (int c0 = 0; c0 < ncand; c0 += 32) {
            const int cnd = c0 + lane;
            const int dcx = cnd % nxc - g.Rx, dcy = cnd / nxc - g.Ry;
            int jx = cx + dcx, jy = cy + dcy;
            const int sx = jx < 0 ? -1 : (jx >= g.ncx ? 1 : 0);
            const int sy = jy < 0 ? -1 : (jy >= g.ncy ? 1 : 0);
            jx -= sx * g.ncx;
            jy -= sy * g.ncy;
            const float cxl = (float)(jx * g.colw[0] + sx * g.L[0]), cxh = (float)((jx + 1) * g.colw[0] + sx * g.L[0]);
            const float cyl = (float)(jy * g.colw[1] + sy * g.L[1]), cyh = (float)((jy + 1) * g.colw[1] + sy * g.L[1]);
            const float gx = fmaxf(0.f, fmaxf(cxl - hi.x, lo.x - cxh));
            const float gy = fmaxf(0.f, fmaxf(cyl - hi.y, lo.y - cyh));
            const int jcol = jy + g.ncy * jx;
            const bool near = cnd < ncand && jcol >= col && gx * gx + gy * gy <= g.rlist2;
            const int j0 = near ? col_cstart[jcol] : 0, j1 = near ? col_cstart[jcol + 1] : 0;
            for (int sz = -1; sz <= 1; ++sz) {
                const float zmin = lo.z - g.rlist - sz * Lz, zmax = hi.z + g.rlist - sz * Lz;
                if (zmax < -1.0f || zmin > Lz + 1.0f) continue;   // the same for every lane
                // the column's clusters are z-sorted: first with hi.z >= zmin, first after it with lo.z > zmax
                int a = j0, b = j1;
                while (a < b) {
                    const int mid = (a + b) >> 1;
                    if (bb_hi[mid].z < zmin) a = mid + 1;
                    else b = mid;
                }
                int e = a;
                b = j1;
                while (e < b) {
                    const int mid = (e + b) >> 1;
                    if (bb_lo[mid].z > zmax) b = mid;
                    else e = mid + 1;
                }
                if (jcol == col) a = max(a, min(I, e));   // j >= i
                int incl = e - a;
                const int len = incl;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += v;
                }
                const int total = __shfl_sync(FULL, incl, 31);
                const int first = a - (incl - len);                // J = first(source lane) + index
                const int img = (sx + 1) + 3 * (sy + 1);
                for (int t0 = 0; t0 < total; t0 += 32) {
                    const int t = t0 + lane;
                    int src = 0;                                   // lanes whose runs end at or before t
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const int v = __shfl_sync(FULL, incl, src + o - 1);
                        if (v <= t) src += o;
                    }
                    const int J = __shfl_sync(FULL, first, src) + t, im = __shfl_sync(FULL, img, src);
                    bool hit = t < total;
                    const int code = im + 9 * (sz + 1);
                    if (hit) {
                        const float4 jl = bb_lo[J], jh = bb_hi[J];
                        const float ox = (im % 3 - 1) * Lx, oy = (im / 3 - 1) * Ly, oz = sz * Lz;
                        const float dx = fmaxf(0.f, fmaxf(jl.x + ox - hi.x, lo.x - (jh.x + ox)));
                        const float dy = fmaxf(0.f, fmaxf(jl.y + oy - hi.y, lo.y - (jh.y + oy)));
                        const float dz = fmaxf(0.f, fmaxf(jl.z + oz - hi.z, lo.z - (jh.z + oz)));
                        hit = dx * dx + dy * dy + dz * dz <= g.rlist2 && !(J < I || (J == I && code < 13));
                    }
                    emit(__ballot_sync(FULL, hit), ((unsigned)J << 5) | (unsigned)code);
                }
            }
        }
    };
    // Masks of the cnt buffered entries, exclusions cleared, written at out[pos0 ..].
    auto finish = [&](int cnt, long long pos0) {
        __syncwarp();
        for (int k = lane; k < cnt; k += 32) {
            const int J = (int)(key[k] >> 5), code = (int)(key[k] & 31u);
            const unsigned long long m = entry_mask(nvi, (int)bb_lo[J].w, J == I && code == 13);
            mask[2 * k] = (unsigned)m;
            mask[2 * k + 1] = (unsigned)(m >> 32);
        }
        __syncwarp();
        const int la = lane >> 2, atom = slot_atom[I * CLUSTER + la];   // four lanes per i atom
        int p = 0, pe = 0;
        if (ex_off && atom >= 0) {
            p = ex_off[atom] + (lane & 3);
            pe = ex_off[atom + 1];
        }
        while (__any_sync(FULL, p < pe)) {
            unsigned want = ~0u;
            int bit = 0;
            if (p < pe && !excluded_entry(I, la, atom, ex_nb[p], atom_slot, xyz, center, g.L, want, bit)) want = ~0u;
            p += 4;
            if (__any_sync(FULL, want != ~0u))
                for (int k = 0; k < cnt; ++k)
                    if (key[k] == want) atomicAnd(&mask[2 * k + (bit >> 5)], ~(1u << (bit & 31)));
        }
        __syncwarp();
        for (int k = lane; k < cnt; k += 32) {
            const long long pos = pos0 + k;
            if (pos >= cap) continue;
            PairEntry e;
            e.j = (int)(key[k] >> 5);
            e.shift = (int)(key[k] & 31u);
            e.mask = ((unsigned long long)mask[2 * k + 1] << 32) | mask[2 * k];
            out[pos] = e;
        }
        __syncwarp();
    };

    int n = 0;
    generate([&](unsigned m, unsigned kk) {
        const int pos = n + __popc(m & below);
        if (((m >> lane) & 1u) && pos < SEARCH_CAP) key[pos] = kk;
        n += __popc(m);
    });
    int start = 0;
    if (lane == 0) {
        start = atomicAdd(d_total, n);
        ILRange r;
        r.i = I;
        r.start = start;
        r.count = n;
        r.pad = 0;
        ilist[I] = r;
        if ((long long)start + n > cap) status_set(st, ST_CAPACITY_PAIRS);
    }
    start = __shfl_sync(FULL, start, 0);
    if (n <= SEARCH_CAP) {
        finish(n, start);
        return;
    }
    int held = 0;
    long long done = start;
    __syncwarp();   // the first pass filled the buffer too
    generate([&](unsigned m, unsigned kk) {
        if (held + __popc(m) > SEARCH_CAP) {
            finish(held, done);
            done += held;
            held = 0;
        }
        if ((m >> lane) & 1u) key[held + __popc(m & below)] = kk;
        held += __popc(m);
    });
    finish(held, done);
}

// Clear the mask bits of listed excluded pairs (those that the search left), a
// warp per pair: its lanes scan the range of the pair's i cluster.
__global__ void __launch_bounds__(256) k_exclusion_masks(int n, const int* __restrict__ pairs, const SearchGeom g,
                                                         const int* __restrict__ atom_slot,
                                                         const double* __restrict__ xyz,
                                                         const double4* __restrict__ center,
                                                         const ILRange* __restrict__ ilist, PairEntry* __restrict__ plist,
                                                         long long cap)
{
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= n) return;
    int a = pairs[2 * k], b = pairs[2 * k + 1];   // a < b
    if (atom_slot[b] / CLUSTER < atom_slot[a] / CLUSTER) {
        const int t = a;
        a = b;
        b = t;
    }
    const int I = atom_slot[a] / CLUSTER;
    unsigned key;
    int bit;
    if (!excluded_entry(I, atom_slot[a] % CLUSTER, a, b, atom_slot, xyz, center, g.L, key, bit)) return;
    const ILRange r = ilist[I];
    const long long end = min((long long)r.start + r.count, cap);
    for (long long e0 = r.start; e0 < end; e0 += 32) {
        const long long e = e0 + lane;
        const bool hit = e < end && plist[e].j == (int)(key >> 5) && plist[e].shift == (int)(key & 31u);
        if (hit) atomicAnd(&plist[e].mask, ~(1ull << bit));
        if (__any_sync(0xffffffffu, hit)) return;
    }
}

// ------------------------------------------------------------- pruning
// Dynamic pruning: keep the outer-list entries that have at least one atom
// pair within the prune radius at the current positions, in list order, packed
// from the i cluster's start offset in the outer list.  The test ignores the
// entry's exclusion mask (an entry whose only close pairs are excluded is
// kept; the pair kernel applies the mask), so it keeps a superset of the exact
// set, and it runs in FP32 in both precisions: |a - b|^2 = |a|^2 + |b|^2 - 2 a.b
// rounds with the square of the clusters' extents, by at most 16 roundings of
// |x|^2: ~1e-4 A^2 at liquid density and 0.05 A^2 at half extents of 128 A, inside
// the radius' 0.02 A margin (0.4 A^2 at a cutoff of 10 A, 0.1 at 3 A).  Wider
// clusters, those of very dilute systems, would lose pairs near the cutoff: where
// there are some, their entries are tested without the expansion, in the
// precision of the positions (WIDE, prune_wide).
//
// W warps share an i cluster (32 entries each per round).  An entry is first
// tested lane by lane through the clusters' current boxes (k_pack): farther
// apart than the radius - dropped; so close that two face atoms must lie
// within it - kept.  The others go to shared memory and are tested eight at a
// time, four lanes each with two j atoms against the eight i atoms in
// registers as packed FP32x2 pairs (three FMAs per two pairs, one three-input
// minimum).
//
// What bounds it: gathers and latency (half the issue slots used, 470 warp
// instructions per 32 entries).  One lane per entry with early exit reads 32
// lines per load instruction and three 16-byte box words per entry; here a box is
// one 16-byte word and a test reads eight whole lines.  FP32 at 100k atoms 44 us
// against 48, at 960k 359 against 408; FP64 half lists at 100k 50 us against 125
// with FP64 arithmetic.  Loading the next 32 entries and
// boxes a round ahead gained nothing (42-52 us); at three blocks per SM,
// without the 48 spilled bytes, 100k took 42 us but 960k 396 us.
using F32x2 = unsigned long long;   // two packed FP32 values
__device__ __forceinline__ F32x2 pack2(float lo, float hi)
{
    F32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c)
{
    F32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float min_with2(float m, F32x2 v)   // min(m, v.lo, v.hi)
{
    float lo, hi, r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(lo), "f"(hi));
    return r;
}

constexpr int PRUNE_WARPS = 8;   // largest block

// One entry without the expansion: bit h set when half h of the i cluster has an
// atom pair within the radius.  Called for clusters too wide for the FP32 test;
// not inlined, so that it takes no registers from it.
template <typename R>
__device__ __noinline__ unsigned prune_wide(const typename V4<R>::type* __restrict__ xi,
                                            const typename V4<R>::type* __restrict__ xj, float ox, float oy, float oz,
                                            float rc2)
{
    unsigned near = 0;
    for (int j = 0; j < CLUSTER && near != 3u; ++j) {
        const typename V4<R>::type b = xj[j];
        const R qx = b.x + ox, qy = b.y + oy, qz = b.z + oz;
        for (int i = 0; i < CLUSTER; ++i) {
            const typename V4<R>::type a = xi[i];
            const R dx = a.x - qx, dy = a.y - qy, dz = a.z - qz;
            if (fma(dx, dx, fma(dy, dy, dz * dz)) < rc2) near |= 1u << (i / 4);
        }
    }
    return near;
}

// HALF: the half layout (4 x 8).  Each half of the i cluster (atoms 0-3, 4-7)
// is tested on its own and an entry goes to the list of every half that has an
// atom pair within the radius.  The outer range [start, start + count) of i
// cluster I owns the slots [2 start + h count, 2 start + (h + 1) count) of the
// half list; item 2 w + h of this launch describes half h (ILRange.pad = h).
template <int W, bool HALF, bool WIDE>
__device__ __forceinline__ void prune_dev(const PruneArgs& A)
{
    // self-pruning: the list pruned last time still holds every pair within the cutoff
    if (!A.force && __uint_as_float(*A.disp) <= A.disp_thr2) return;
    __shared__ float sh[27][6];
    __shared__ float4 cand[PRUNE_WARPS][32];          // the entries to test: J's frame origin seen from I's, J
    __shared__ unsigned kmask[2][HALF ? 2 : 1][W];    // kept entries of a round, per warp of the cluster (W > 1)
    for (int k = threadIdx.x; k < 27 * 6; k += blockDim.x) sh[k / 6][k % 6] = A.shifts.v[k / 6][k % 6];
    __syncthreads();
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // W == 1: the block's warps take a cluster each; W > 1: a block of W warps takes one
    const int w = W == 1 ? (int)(blockIdx.x * (blockDim.x >> 5)) + wib : (int)blockIdx.x;
    const int sub = W == 1 ? 0 : wib;
    if (w >= A.ncl) return;
    const unsigned below = (1u << lane) - 1u;
    const ILRange L = A.ilist[w];
    const int I = L.i;
    const float4* __restrict__ xf = A.xf;
    if (sub == 0 && lane < CLUSTER) {
        if (A.snap_d) A.snap_d[I * CLUSTER + lane] = A.xd[I * CLUSTER + lane];
        else if (A.snap_f) A.snap_f[I * CLUSTER + lane] = xf[I * CLUSTER + lane];
    }
    F32x2 ax[4], ay[4], az[4], an[4];   // -2 x_i and |x_i|^2 of atoms 2k, 2k + 1
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 u = xf[I * CLUSTER + 2 * k], v = xf[I * CLUSTER + 2 * k + 1];
        ax[k] = pack2(-2.f * u.x, -2.f * v.x);
        ay[k] = pack2(-2.f * u.y, -2.f * v.y);
        az[k] = pack2(-2.f * u.z, -2.f * v.z);
        an[k] = pack2(u.x * u.x + u.y * u.y + u.z * u.z, v.x * v.x + v.y * v.y + v.z * v.z);
    }
    const float4 cI = A.centerf[I];
    const BoxF bi = box_decode(A.box[I]);
    const float rc2 = A.rcut2;
    const long long out0 = HALF ? 2LL * L.start : L.start, out1 = 2LL * L.start + L.count;
    int kept0 = 0, kept1 = 0, buf = 0;
    for (int base = 0; base < L.count; base += 32 * W) {
        const int e = base + 32 * sub + lane;
        const bool have = e < L.count;
        PairEntry my;
        my.j = I; my.shift = 13; my.mask = 0ull;
        if (have) my = A.plist[L.start + e];
        const BoxF bj = box_decode(A.box[my.j]);
        const float* s6 = sh[my.shift];
        const float dx = fabsf((bi.x - bj.x) - s6[0]), dy = fabsf((bi.y - bj.y) - s6[1]),
                    dz = fabsf((bi.z - bj.z) - s6[2]);
        const float sx = bi.hx + bj.hx, sy = bi.hy + bj.hy, sz = bi.hz + bj.hz;
        const float gx = fmaxf(0.f, dx - sx), gy = fmaxf(0.f, dy - sy), gz = fmaxf(0.f, dz - sz);
        bool todo = have && my.mask != 0ull && gx * gx + gy * gy + gz * gz < rc2;
        bool k0 = false, k1 = false;
        if (!HALF) {
            // the face atoms towards each other along one axis: that far apart
            // along it (+ the boxes' padding and their rounding to 1/64 A), at most the spans along the others
            const float ux = fabsf(dx - sx) + 0.04f, uy = fabsf(dy - sy) + 0.04f, uz = fabsf(dz - sz) + 0.04f;
            const float wx = (dx + sx) * (dx + sx), wy = (dy + sy) * (dy + sy), wz = (dz + sz) * (dz + sz);
            const float far2 = fminf(ux * ux + wy + wz, fminf(wx + uy * uy + wz, wx + wy + uz * uz));
            k0 = todo && far2 < rc2 && A.box_fine && bi.fine && bj.fine;
            todo = todo && !k0;
        }
        if (WIDE && todo &&
            fmaxf(fmaxf(fmaxf(bi.hx, bi.hy), fmaxf(bi.hz, bj.hx)), fmaxf(bj.hy, bj.hz)) > 0.5f * WIDE_EXTENT) {
            const float4 cJ = A.centerf[my.j];
            const float ox = -(((cI.x - cJ.x) - s6[0]) - s6[3]), oy = -(((cI.y - cJ.y) - s6[1]) - s6[4]),
                        oz = -(((cI.z - cJ.z) - s6[2]) - s6[5]);
            const size_t si = (size_t)I * CLUSTER, sj = (size_t)my.j * CLUSTER;
            const unsigned near = A.xd ? prune_wide<double>(A.xd + si, A.xd + sj, ox, oy, oz, rc2)
                                       : prune_wide<float>(xf + si, xf + sj, ox, oy, oz, rc2);
            k0 = HALF ? (near & 1u) != 0u : near != 0u;
            k1 = HALF && (near & 2u) != 0u;
            todo = false;
        }
        const unsigned tb = __ballot_sync(0xffffffffu, todo);
        const int rank = __popc(tb & below), n = __popc(tb);
        if (todo) {
            const float4 cJ = A.centerf[my.j];
            cand[wib][rank] = make_float4(-(((cI.x - cJ.x) - s6[0]) - s6[3]), -(((cI.y - cJ.y) - s6[1]) - s6[4]),
                                          -(((cI.z - cJ.z) - s6[2]) - s6[5]), __int_as_float(my.j));
        }
        __syncwarp();
        for (int p = 0; p < n; p += 8) {
            const float4 o = cand[wib][min(p + (lane >> 2), n - 1)];
            const float4* __restrict__ xj = xf + (size_t)__float_as_int(o.w) * CLUSTER + 2 * (lane & 3);
            float4 v[2];
            v[0] = xj[0];
            v[1] = xj[1];
            bool h0 = false, h1 = false;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float qx = v[u].x + o.x, qy = v[u].y + o.y, qz = v[u].z + o.z;
                const float thr = rc2 - (qx * qx + qy * qy + qz * qz);
                const F32x2 qx2 = pack2(qx, qx), qy2 = pack2(qy, qy), qz2 = pack2(qz, qz);
                float m0 = 3.0e38f, m1 = 3.0e38f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const F32x2 d = fma2(ax[k], qx2, fma2(ay[k], qy2, fma2(az[k], qz2, an[k])));
                    if (HALF && k >= 2) m1 = min_with2(m1, d);
                    else m0 = min_with2(m0, d);
                }
                h0 = h0 || m0 < thr;
                if (HALF) h1 = h1 || m1 < thr;
            }
            const unsigned b0 = __ballot_sync(0xffffffffu, h0), b1 = HALF ? __ballot_sync(0xffffffffu, h1) : 0u;
            if (todo && (rank >> 3) == (p >> 3)) {
                k0 = ((b0 >> (4 * (rank & 7))) & 0xfu) != 0u;
                if (HALF) k1 = ((b1 >> (4 * (rank & 7))) & 0xfu) != 0u;
            }
        }
        const unsigned m0 = __ballot_sync(0xffffffffu, k0), m1 = HALF ? __ballot_sync(0xffffffffu, k1) : 0u;
        int off0 = kept0, off1 = kept1;
        if (W == 1) {
            kept0 += __popc(m0);
            kept1 += __popc(m1);
        } else {
            if (lane == 0) {
                kmask[buf][0][sub] = m0;
                if (HALF) kmask[buf][HALF ? 1 : 0][sub] = m1;
            }
            __syncthreads();   // every warp of the block runs the same rounds
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const int c0 = __popc(kmask[buf][0][k]), c1 = HALF ? __popc(kmask[buf][HALF ? 1 : 0][k]) : 0;
                if (k < sub) {
                    off0 += c0;
                    off1 += c1;
                }
                kept0 += c0;
                kept1 += c1;
            }
            buf ^= 1;   // the other buffer next round: no second barrier
        }
        if (k0) A.plist_in[out0 + off0 + __popc(m0 & below)] = my;
        if (HALF && k1) A.plist_in[out1 + off1 + __popc(m1 & below)] = my;
    }
    if (lane == 0 && sub == 0) {
        ILRange r;
        r.i = I; r.start = (int)out0; r.count = kept0; r.pad = 0;
        A.ilist_in[HALF ? 2 * w : w] = r;
        if (HALF) {
            r.start = (int)out1; r.count = kept1; r.pad = 1;
            A.ilist_in[2 * w + 1] = r;
        }
    }
}

template <int W, bool HALF, bool WIDE>
__global__ void __launch_bounds__(W == 1 ? 256 : 32 * W, W == 1 ? 4 : 32 / W) k_prune(PruneArgs A)
{
    prune_dev<W, HALF, WIDE>(A);
}

template <int W, bool HALF, bool WIDE>
__global__ void __launch_bounds__(W == 1 ? 256 : 32 * W, W == 1 ? 4 : 32 / W)
    k_prune_multi(const PruneArgs* __restrict__ As)
{
    const PruneArgs& A = As[blockIdx.z];
    if ((int)blockIdx.x >= A.gx) return;
    prune_dev<W, HALF, WIDE>(A);
}

// Warps per i cluster of a launch over ncl clusters: four where one each
// leaves SMs idle.  2,780 atoms (372 clusters) 24 -> 14 us, 7,309 atoms (941)
// 21 -> 14 us; at 3,241 clusters 25 -> 21 us alone, but the evaluation went
// from 130 to 135 us (the side stream fills the idle issue slots), and at
// 12,144 the prune itself from 44 to 57 us.
void set_prune_warps(PruneArgs& A, long long ncl)
{
    A.warps = ncl < 2048 ? 4 : 1;
    A.gx = A.warps == 1 ? grid_blocks((long long)A.ncl * 32, 256) : std::max(1, A.ncl);
}

// Padding of the boxes against the FP32 rounding of their absolute centres
// and of the image offsets: 4e-7 of the longest edge covers it.
static float box_pad(const Ctx& c)
{
    return 1e-3f + 4e-7f * (float)std::max(c.box[0], std::max(c.box[1], c.box[2]));
}

// Prune arguments for this rank's i clusters (ncl = 0: nothing to do);
// half: write the half lists (item 2 w + h of this rank's range).
PruneArgs make_prune_args(const Ctx& c, bool half)
{
    PruneArgs A;
    // a hair above the cutoff so FP32 rounding never drops a pair at r ~ rc
    const double rc = c.p.cutoff + std::max(0.0, c.p.prune_margin) + 0.02;
    A.shifts = make_shift_table(c);
    long long lo, hi;
    cluster_share(c, lo, hi);   // this rank's i clusters
    A.ncl = (int)(hi - lo);
    A.gy = 1;
    set_prune_warps(A, A.ncl);
    A.ilist = c.ilist.p + lo;
    A.plist = c.plist.p;
    A.xf = c.xq_f.p;
    A.xd = c.xq_d.p;
    A.centerf = c.centerf.p;
    A.box = c.cur_box.p;
    A.box_fine = box_pad(c) < 0.002f ? 1 : 0;
    A.rcut2 = (float)(rc * rc);
    A.ilist_in = half ? c.ilist_h.p + 2 * lo : c.ilist_in.p + lo;
    A.plist_in = half ? c.plist_h.p : c.plist_in.p;
    const bool selfp = self_pruning(c), mixed = c.p.precision == MDF_PREC_MIXED;
    A.snap_f = selfp && mixed ? reinterpret_cast<float4*>(c.xq_snap.p) : nullptr;
    A.snap_d = selfp && !mixed ? reinterpret_cast<double4*>(c.xq_snap.p) : nullptr;
    A.disp = reinterpret_cast<const unsigned*>(c.scal.p + SCAL_DISP);
    const float half_margin = (float)(0.5 * std::max(0.0, c.p.prune_margin));
    A.disp_thr2 = half_margin * half_margin;
    A.force = (!selfp || !c.pruned_valid) ? 1 : 0;
    return A;
}

// The half-layout lists (two items per i cluster, twice the outer capacity).
void ensure_half_lists(Ctx& c)
{
    c.ilist_h.alloc(2 * (size_t)std::max(c.n_clusters, 1));
    c.plist_h.alloc(2 * (size_t)std::max<size_t>(c.plist.n, 1));
}

// A prune kernel's launch.  A self-pruning one mostly returns at once, but an SM
// has to drain to change how much of its L1 is shared memory, and the driver's
// choice for this kernel differs from the pair kernel's: asking for the pair
// kernel's (72% of the L1, three blocks) took a step of 28k-atom dynamics from
// 130 to 121 us.  A prune that does the work keeps the driver's choice, whose
// larger L1 it needs (100k atoms 44 against 48 us).
template <typename A>
static void launch_prune(void (*kern)(A), A arg, dim3 grid, int threads, bool selfp, cudaStream_t s)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = 72;
    cfg.attrs = &at;
    cfg.numAttrs = selfp ? 1 : 0;
    MDF_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, arg));
}

// The prune kernel of a form: single system (PruneArgs) or many (const PruneArgs*).
template <bool WIDE>
static auto prune_kernel(int warps, bool half) -> void (*)(PruneArgs)
{
    if (warps == 1) return half ? k_prune<1, true, WIDE> : k_prune<1, false, WIDE>;
    return half ? k_prune<4, true, WIDE> : k_prune<4, false, WIDE>;
}
template <bool WIDE>
static auto prune_kernel_multi(int warps, bool half) -> void (*)(const PruneArgs*)
{
    if (warps == 1) return half ? k_prune_multi<1, true, WIDE> : k_prune_multi<1, false, WIDE>;
    return half ? k_prune_multi<4, true, WIDE> : k_prune_multi<4, false, WIDE>;
}

// warps: the same in every system's arguments; wide: some system has wide clusters.
void launch_prune_multi(const PruneArgs* d_args, int nsys, int gx, int warps, bool half, bool wide, bool selfp,
                        cudaStream_t s)
{
    launch_prune<const PruneArgs*>(wide ? prune_kernel_multi<true>(warps, half) : prune_kernel_multi<false>(warps, half),
                                   d_args, dim3(gx, 1, nsys), warps == 1 ? 256 : 128, selfp, s);
}

// whole_entries: build the 8 x 8 pruned list even in the half layout (the
// adjoint walks whole entries); it also prunes unconditionally.
void prune_pairlist(Ctx& c, bool whole_entries)
{
    if (whole_entries) c.pruned_valid = false;   // a self-pruning launch prunes when the list is not valid
    const bool half = half_layout(c) && !whole_entries;
    if (half) ensure_half_lists(c);
    const PruneArgs A = make_prune_args(c, half);
    if (A.ncl > 0)
        launch_prune<PruneArgs>(c.wide_clusters ? prune_kernel<true>(A.warps, half) : prune_kernel<false>(A.warps, half),
                                A, grid_of(A), A.warps == 1 ? 256 : 128, !A.force, c.stream);
    c.launches += 1;
    c.pruned_valid = true;
    c.pruned_half = half;
}

// ------------------------------------------------------------------ host
static double atom_density(const Ctx& c)
{
    return (double)c.N / (c.box[0] * c.box[1] * c.box[2]);
}

template <typename R>
PackArgs<R> make_pack_args(const Ctx& c)
{
    PackArgs<R> A;
    A.nslots = c.n_slots;
    A.gx = grid_blocks(c.n_slots, 256);
    A.gy = 1;
    A.xyz = c.xyz.p;
    A.q = c.q.p;
    A.slot_atom = c.slot_atom.p;
    A.center = c.center.p;
    for (int d = 0; d < 3; ++d) A.L[d] = c.box[d];
    A.xq = reinterpret_cast<typename V4<R>::type*>(sizeof(R) == 4 ? (void*)c.xq_f.p : (void*)c.xq_d.p);
    A.box = c.cur_box.p;
    A.box_pad = box_pad(c);
    A.xf = c.xq_f.p;
    A.snap = self_pruning(c) ? reinterpret_cast<const typename V4<R>::type*>(c.xq_snap.p) : nullptr;
    A.disp = reinterpret_cast<unsigned*>(c.scal.p + SCAL_DISP);
    A.st = c.status.p;
    return A;
}
template PackArgs<float> make_pack_args<float>(const Ctx&);
template PackArgs<double> make_pack_args<double>(const Ctx&);

template <typename R>
void launch_pack_multi(const PackArgs<R>* d_args, BlockMap bm, cudaStream_t s)
{
    if (bm.n <= 0) return;
    k_pack_multi<R><<<bm.n, 256, 0, s>>>(d_args, bm.map);
    MDF_CUDA_TRY(cudaGetLastError());
}
template void launch_pack_multi<float>(const PackArgs<float>*, BlockMap, cudaStream_t);
template void launch_pack_multi<double>(const PackArgs<double>*, BlockMap, cudaStream_t);

void pack_positions(Ctx& c)
{
    if (c.p.precision == MDF_PREC_MIXED) {
        const PackArgs<float> A = make_pack_args<float>(c);
        k_pack<float><<<grid_of(A), 256, 0, c.stream>>>(A);
    } else {
        const PackArgs<double> A = make_pack_args<double>(c);
        k_pack<double><<<grid_of(A), 256, 0, c.stream>>>(A);
    }
    MDF_CUDA_TRY(cudaGetLastError());
    c.launches += 1;
}

// Bands of a split evaluation (the arithmetic in bands.hpp): this rank's
// clusters, its stencil window and its halo plane lists, uploaded once per
// build.
void build_bands(Ctx& c)
{
    const int P = c.p.nranks, me = c.p.rank, K0 = c.K[0];
    const int ncy = c.ncol_y;
    std::vector<int> cst(c.ncols + 1);
    MDF_CUDA_TRY(cudaMemcpyAsync(cst.data(), c.col_cstart.p, sizeof(int) * (c.ncols + 1), cudaMemcpyDeviceToHost,
                                 c.stream));
    MDF_CUDA_TRY(cudaStreamSynchronize(c.stream));
    const BandPlan B = plan_bands(P, K0, c.ncol_x, c.box[0], c.p.skin);
    c.band_cl.assign(P + 1, 0);
    for (int t = 0; t <= P; ++t) c.band_cl[t] = cst[B.first[t] * ncy];
    c.win_lo = B.win_lo;
    c.win_n = B.win_n;
    const HaloLists H = halo_lists(B, P, me, K0);
    auto upload = [&](DevBuf<int>& d, const std::vector<int>& h) {
        d.alloc(std::max<size_t>(1, h.size()));
        if (!h.empty())
            MDF_CUDA_TRY(cudaMemcpyAsync(d.p, h.data(), sizeof(int) * h.size(), cudaMemcpyHostToDevice, c.stream));
    };
    upload(c.halo_send_pl, H.send);
    upload(c.halo_recv_pl, H.recv);
    upload(c.halo_local_pl, H.local);
    c.halo_send_n = H.send_n;
    c.halo_recv_n = H.recv_n;
    c.halo_n_send = (int)H.send.size();
    c.halo_n_recv = (int)H.recv.size();
    c.halo_n_local = (int)H.local.size();
    for (int k = 0; k < 2; ++k)
        for (int l = 0; l < 2; ++l) c.halo_rng[k][l] = H.rng[k][l];
    MDF_CUDA_TRY(cudaStreamSynchronize(c.stream));   // the host lists are freed on return
}


// The whole build is queued on the context's stream without a host round trip
// in between: every buffer the build kernels write is sized from bounds known
// on the host (clusters <= ceil(N/8) + columns; the list from a density
// estimate or the last build), the kernels read the cluster count from the
// device, and one synchronisation at the end returns the cluster and entry
// counts with the status word.  A list that outgrew its capacity is grown and
// searched again; a column above the sort's limit restarts with thinner
// columns.
void build_pairlist(Ctx& c)
{
    c.npairs_dev.alloc(1);
    c.count_next = true;
    c.counted = false;
    cudaStream_t s = c.stream;
    const int th = 256;
    const double rlist = c.p.cutoff + c.p.skin;
    for (int d = 0; d < 3; ++d)
        if (!(c.box[d] >= 2.0 * c.p.cutoff))
            throw ApiError(MDF_ERR_INVALID, "box edge shorter than twice the cutoff (minimum image undefined)");
    if (!c.h_build) MDF_CUDA_TRY(cudaHostAlloc((void**)&c.h_build, 4 * sizeof(int), cudaHostAllocDefault));
    c.d_build.alloc(4);
    // column cross-section ~ one cluster of atoms per column-height cube
    const double rho = atom_density(c);
    double side = std::cbrt((double)CLUSTER / std::max(rho, 1e-6));
    for (int attempt = 0; attempt < 6; ++attempt) {
        c.ncol_x = std::max(1, (int)std::floor(c.box[0] / side));
        c.ncol_y = std::max(1, (int)std::floor(c.box[1] / side));
        // The one-image search visits the +-R columns around a column (R =
        // floor(rlist / width) + 1), which must be distinct: R < columns.
        // Sparse systems start from wide columns; add columns until it holds.
        auto reach = [&](double L, int nc) { return (int)std::floor(rlist / (L / nc)) + 1; };
        while (reach(c.box[0], c.ncol_x) >= c.ncol_x && c.ncol_x < 4096) ++c.ncol_x;
        while (reach(c.box[1], c.ncol_y) >= c.ncol_y && c.ncol_y < 4096) ++c.ncol_y;
        const int Rx = reach(c.box[0], c.ncol_x), Ry = reach(c.box[1], c.ncol_y);
        if (Rx >= c.ncol_x || Ry >= c.ncol_y) throw ApiError(MDF_ERR_INVALID, "box too small for the list cutoff");
        c.ncols = c.ncol_x * c.ncol_y;
        // every column wastes at most one partly filled cluster
        const long long ncl_cap = ((long long)c.N + CLUSTER - 1) / CLUSTER + c.ncols;
        if (ncl_cap * CLUSTER > INT32_MAX / 3) throw ApiError(MDF_ERR_CAPACITY, "too many atoms for one context");
        c.col_count.alloc(c.ncols + 1);
        c.col_start.alloc(c.ncols + 1);
        c.col_cstart.alloc(c.ncols + 1);
        c.atom_col.alloc(c.N);   // (column, place in it)
        c.col_atoms.alloc(c.N);
        c.atom_slot.alloc(c.N);
        c.slot_atom.alloc(ncl_cap * CLUSTER);
        c.slot_type.alloc(ncl_cap * CLUSTER);
        c.cluster_col.alloc(ncl_cap);
        c.center.alloc(ncl_cap);
        c.centerf.alloc(ncl_cap);
        c.bb_lo.alloc(ncl_cap);
        c.bb_hi.alloc(ncl_cap);
        c.ilist.alloc(ncl_cap);
        if (!c.plist.p) {
            // list estimate: half the clusters within rlist + one cluster extent, 30% over
            const double ext = rlist + side;
            const double per = 0.5 * (rho / CLUSTER) * (4.0 / 3.0) * M_PI * ext * ext * ext * 1.3;
            c.plist.alloc((size_t)(ncl_cap * std::max(32.0, per)) + 1024);
        }
        {
            // largest power-of-two quantum keeping every centre exact in FP32 (24-bit significand)
            const double lmax = std::max(c.box[0], std::max(c.box[1], c.box[2]));
            c.center_quantum = std::ldexp(1.0, (int)std::ceil(std::log2(lmax + 1.0)) - 24);
        }
        const int* d_ncl = c.col_cstart.p + c.ncols;   // cluster count, written by k_column_table
        MDF_CUDA_TRY(cudaMemsetAsync(c.col_count.p, 0, sizeof(int) * (c.ncols + 1), s));
        MDF_CUDA_TRY(cudaMemsetAsync(c.status.p, 0, sizeof(unsigned), s));
        k_assign_columns<<<grid_blocks(c.N, th), th, 0, s>>>(c.N, c.xyz.p, c.box[0], c.box[1], c.ncol_x, c.ncol_y,
                                                             c.atom_col.p, c.col_count.p, c.status.p);
        k_column_table<<<1, 1024, 0, s>>>(c.ncols, c.col_count.p, c.col_start.p, c.col_cstart.p, c.status.p);
        k_bucket<<<grid_blocks(c.N, th), th, 0, s>>>(c.N, c.atom_col.p, c.col_start.p, c.col_atoms.p);
        k_sort_columns<<<c.ncols, SORT_THREADS, 0, s>>>(c.xyz.p, c.box[2], c.col_count.p, c.col_start.p, c.col_cstart.p,
                                                c.col_atoms.p, c.slot_atom.p, c.atom_slot.p, c.cluster_col.p,
                                                c.status.p);
        k_cluster_geom<<<grid_blocks(ncl_cap * CLUSTER, th), th, 0, s>>>(
            d_ncl, c.xyz.p, c.box[0], c.box[1], c.box[2], c.center_quantum, c.slot_atom.p, c.type.p, c.ntp - 1,
            c.center.p, c.centerf.p, c.bb_lo.p, c.bb_hi.p, c.slot_type.p);
        MDF_CUDA_TRY(cudaGetLastError());

        SearchGeom g;
        for (int d = 0; d < 3; ++d) g.L[d] = c.box[d];
        g.colw[0] = c.box[0] / c.ncol_x;
        g.colw[1] = c.box[1] / c.ncol_y;
        g.colw[2] = c.box[2];
        g.ncx = c.ncol_x;
        g.ncy = c.ncol_y;
        g.Rx = Rx;
        g.Ry = Ry;
        // bounding boxes are rounded outward to float; pad the list radius a hair
        g.rlist = (float)(rlist * (1.0 + 1e-6));
        g.rlist2 = g.rlist * g.rlist;
        unsigned st = 0;
        for (int search = 0; search < 3; ++search) {
            const long long cap = (long long)c.plist.n;
            MDF_CUDA_TRY(cudaMemsetAsync(c.d_build.p, 0, sizeof(int) * 4, s));
            k_pair_search<<<grid_blocks(ncl_cap, SEARCH_WARPS), 32 * SEARCH_WARPS, 0, s>>>(
                d_ncl, g, c.cluster_col.p, c.col_cstart.p, c.bb_lo.p, c.bb_hi.p, c.center.p, c.slot_atom.p,
                c.atom_slot.p, c.xyz.p, c.n_excl > 0 ? c.ex_rows.p : nullptr,
                c.n_excl > 0 ? c.ex_rows.p + c.N + 1 : nullptr, c.d_build.p, c.plist.p, cap, c.ilist.p, c.status.p);
            if (c.n_ex_heavy > 0)
                k_exclusion_masks<<<grid_blocks(32LL * c.n_ex_heavy, th), th, 0, s>>>(
                    c.n_ex_heavy, c.ex_heavy.p, g, c.atom_slot.p, c.xyz.p, c.center.p, c.ilist.p, c.plist.p, cap);
            MDF_CUDA_TRY(cudaGetLastError());
            MDF_CUDA_TRY(cudaMemcpyAsync(c.h_build, d_ncl, sizeof(int), cudaMemcpyDeviceToHost, s));
            MDF_CUDA_TRY(cudaMemcpyAsync(c.h_build + 1, c.d_build.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
            MDF_CUDA_TRY(cudaMemcpyAsync(c.h_build + 3, c.status.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
            MDF_CUDA_TRY(cudaStreamSynchronize(s));
            st = (unsigned)c.h_build[3];
            if (st & (ST_NONFINITE | ST_CAPACITY_COLUMN)) break;
            if (!(st & ST_CAPACITY_PAIRS)) break;
            // the list outgrew its buffer: grow to the count found (+1/8) and search again
            c.plist.alloc((size_t)c.h_build[1] + 1);
            MDF_CUDA_TRY(cudaMemsetAsync(c.status.p, 0, sizeof(unsigned), s));
        }
        if (st & ST_NONFINITE) throw ApiError(MDF_ERR_NONFINITE, "non-finite position");
        if (st & ST_CAPACITY_COLUMN) {
            side *= 0.7;   // too many atoms in a column: thinner columns
            if (attempt == 5) throw ApiError(MDF_ERR_CAPACITY, "column too populated for the in-block sort");
            continue;
        }
        if (st & ST_CAPACITY_PAIRS) throw ApiError(MDF_ERR_CAPACITY, "pair list capacity exceeded");
        const int ncl = c.h_build[0];
        c.n_clusters = ncl;
        c.n_slots = ncl * CLUSTER;
        c.n_entries = c.h_build[1];
        c.wide_clusters = c.h_build[2] != 0;
        c.cur_box.alloc(ncl);
        c.xq_f.alloc(c.n_slots);
        if (c.p.precision != MDF_PREC_MIXED) c.xq_d.alloc(c.n_slots);
        if (c.p.prune_every < 0)
            c.xq_snap.alloc((c.p.precision == MDF_PREC_MIXED ? sizeof(float4) : sizeof(double4)) * (size_t)c.n_slots);
        if (half_layout(c)) ensure_half_lists(c);   // sized here, not inside a later stream capture
        c.f_slot.alloc((size_t)3 * c.n_slots);
        c.need_clear = true;   // slot layout changed: clear the accumulators before the next evaluation
        c.plist_in.alloc(c.plist.n);
        c.ilist_in.alloc(ncl);
        c.pruned_valid = false;
        c.since_prune = 0;
        if (distributed(c)) build_bands(c);
        c.have_list = true;
        return;
    }
}

}  // namespace mdf
