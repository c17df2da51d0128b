// FFT passes of lengths with two or three register radices (fft_radices): the
// production path of the reciprocal space; other lengths keep the table-driven
// passes of pme.cu.
//
// What bounds them: on large grids the L2/HBM traffic of one read and one write
// of the half-complex grid per pass, on small ones latency.  A length n = r1 r2
// (or r1 r2 r3, radices up to 12) takes a radix-r butterfly per thread in
// registers: the first stage's loads come straight from the grid, the last
// stage's results go straight back, and between stages the lines cross shared
// memory once - for 100 = 10 x 10 one exchange and one barrier, where the
// 4 x 5 x 5 table-driven pass staged the lines, wrote and read shared memory
// three times and looked up an index per butterfly.  The x pass multiplies by
// the influence function while the last forward stage's results are in
// registers: element j + r n/R of the last radix R is what the first stage of
// an inverse transform with the radices reversed takes, so convolution and
// turn-around need no exchange either. 
//
// 216^3 (960k atoms) a chain 306 -> 165 us, with energies 345 -> 196; 100^3 FP64
// 83 -> 67; 30^3 36 -> 29.  100^3 FP32 alone is latency either way (52 us), but
// takes fewer issue slots from the pair kernel beside it.
#pragma once

#include "kargs.cuh"

namespace mdf {

template <typename R> struct CT;
template <> struct CT<float> { using type = float2; };
template <> struct CT<double> { using type = double2; };

constexpr int FFT_THREADS = 128;

template <typename C>
__device__ __forceinline__ C cmul(C a, C b)
{
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}

// Rounded product, never contracted with an addition: the convolution gives the
// same bits with energies (through shared memory) and without (in registers).
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

template <typename C>
__device__ __forceinline__ C cconj(C a)
{
    a.y = -a.y;
    return a;
}

// cos and sin of 2 pi k/n at compile time (Taylor series around 0 after
// folding into the first octant), for the constant twiddles inside a radix.
constexpr double tau_series(int k, int n, bool want_sin)
{
    const double t = 6.283185307179586476925287 * k / n;
    double term = want_sin ? t : 1.0, sum = term;
    for (int i = 1; i < 30; ++i) {
        const int a = 2 * i - (want_sin ? 0 : 1);
        term *= -t * t / (a * (a + 1.0));
        sum += term;
    }
    return sum;
}
constexpr double cos_tau(int k, int n);
constexpr double sin_tau(int k, int n)
{
    k %= n;
    return 2 * k > n ? -sin_tau(n - k, n) : 4 * k > n ? sin_tau(n - 2 * k, 2 * n) : 8 * k > n ? cos_tau(n - 4 * k, 4 * n)
                                                                                         : tau_series(k, n, true);
}
constexpr double cos_tau(int k, int n)
{
    k %= n;
    return 2 * k > n ? cos_tau(n - k, n) : 4 * k > n ? -cos_tau(n - 2 * k, 2 * n) : 8 * k > n ? sin_tau(n - 4 * k, 4 * n)
                                                                                         : tau_series(k, n, false);
}

template <int N>
struct TauTable {
    double c[N], s[N];
    constexpr TauTable() : c(), s()
    {
        for (int k = 0; k < N; ++k) {
            c[k] = cos_tau(k, N);
            s[k] = sin_tau(k, N);
        }
    }
};

// In-register DFT of N values; forward uses W = exp(-2 pi i / N).
template <int N, bool INV, typename R, typename C>
struct RDft {
    // N = A B by Cooley-Tukey: B transforms of length A, constant twiddles, A transforms of length B
    static constexpr int A = N % 2 == 0 ? (N % 4 == 0 && N != 8 ? 4 : 2) : 3, B = N / A;
    static __device__ __forceinline__ void run(C (&v)[N])
    {
        constexpr TauTable<N> T{};
        C t[B][A];
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int a = 0; a < A; ++a) t[b][a] = v[B * a + b];
            RDft<A, INV, R, C>::run(t[b]);
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
            C u[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                if (a * b == 0) u[b] = t[b][a];
                else {
                    const C w = {(R)T.c[(a * b) % N], (R)(INV ? T.s[(a * b) % N] : -T.s[(a * b) % N])};
                    u[b] = cmul(t[b][a], w);
                }
            }
            RDft<B, INV, R, C>::run(u);
#pragma unroll
            for (int b = 0; b < B; ++b) v[a + A * b] = u[b];
        }
    }
};
template <bool INV, typename R, typename C>
struct RDft<1, INV, R, C> {
    static __device__ __forceinline__ void run(C (&)[1]) {}
};
template <bool INV, typename R, typename C>
struct RDft<2, INV, R, C> {
    static __device__ __forceinline__ void run(C (&v)[2])
    {
        const C a = v[0], b = v[1];
        v[0].x = a.x + b.x; v[0].y = a.y + b.y;
        v[1].x = a.x - b.x; v[1].y = a.y - b.y;
    }
};
template <bool INV, typename R, typename C>
struct RDft<3, INV, R, C> {
    static __device__ __forceinline__ void run(C (&v)[3])
    {
        const R s1 = (INV ? (R)1 : (R)-1) * (R)0.86602540378443864676;
        const C a = v[0], b = v[1], c = v[2];
        const C t = {b.x + c.x, b.y + c.y}, u = {b.x - c.x, b.y - c.y};
        v[0].x = a.x + t.x; v[0].y = a.y + t.y;
        const C m = {a.x - (R)0.5 * t.x, a.y - (R)0.5 * t.y};
        v[1].x = m.x - s1 * u.y; v[1].y = m.y + s1 * u.x;
        v[2].x = m.x + s1 * u.y; v[2].y = m.y - s1 * u.x;
    }
};
template <bool INV, typename R, typename C>
struct RDft<4, INV, R, C> {
    static __device__ __forceinline__ void run(C (&v)[4])
    {
        const C a = v[0], b = v[1], c = v[2], d = v[3];
        const C t0 = {a.x + c.x, a.y + c.y}, t1 = {a.x - c.x, a.y - c.y};
        const C t2 = {b.x + d.x, b.y + d.y}, t3 = {b.x - d.x, b.y - d.y};
        const C t3r = INV ? C{-t3.y, t3.x} : C{t3.y, -t3.x};   // times +-i
        v[0].x = t0.x + t2.x; v[0].y = t0.y + t2.y;
        v[2].x = t0.x - t2.x; v[2].y = t0.y - t2.y;
        v[1].x = t1.x + t3r.x; v[1].y = t1.y + t3r.y;
        v[3].x = t1.x - t3r.x; v[3].y = t1.y - t3r.y;
    }
};
template <bool INV, typename R, typename C>
struct RDft<5, INV, R, C> {
    static __device__ __forceinline__ void run(C (&v)[5])
    {
        const R s = INV ? (R)1 : (R)-1;
        const R c1 = (R)0.30901699437494742410, c2 = (R)-0.80901699437494742410;
        const R s1 = s * (R)0.95105651629515357212, s2 = s * (R)0.58778525229247312917;
        const C a = v[0];
        const C b1 = {v[1].x + v[4].x, v[1].y + v[4].y}, d1 = {v[1].x - v[4].x, v[1].y - v[4].y};
        const C b2 = {v[2].x + v[3].x, v[2].y + v[3].y}, d2 = {v[2].x - v[3].x, v[2].y - v[3].y};
        v[0].x = a.x + b1.x + b2.x; v[0].y = a.y + b1.y + b2.y;
        const C m1 = {a.x + c1 * b1.x + c2 * b2.x, a.y + c1 * b1.y + c2 * b2.y};
        const C m2 = {a.x + c2 * b1.x + c1 * b2.x, a.y + c2 * b1.y + c1 * b2.y};
        const C n1 = {s1 * d1.x + s2 * d2.x, s1 * d1.y + s2 * d2.y};
        const C n2 = {s2 * d1.x - s1 * d2.x, s2 * d1.y - s1 * d2.y};
        v[1].x = m1.x - n1.y; v[1].y = m1.y + n1.x;
        v[4].x = m1.x + n1.y; v[4].y = m1.y - n1.x;
        v[2].x = m2.x - n2.y; v[2].y = m2.y + n2.x;
        v[3].x = m2.x + n2.y; v[3].y = m2.y - n2.x;
    }
};

template <int N> struct RadixTag { static constexpr int value = N; };

// f(RadixTag<r>) for the runtime radix r.
template <typename F>
__device__ __forceinline__ void with_radix(int r, F&& f)
{
    switch (r) {
        case 1: f(RadixTag<1>{}); break;
        case 2: f(RadixTag<2>{}); break;
        case 3: f(RadixTag<3>{}); break;
        case 4: f(RadixTag<4>{}); break;
        case 5: f(RadixTag<5>{}); break;
        case 6: f(RadixTag<6>{}); break;
        case 8: f(RadixTag<8>{}); break;
        case 9: f(RadixTag<9>{}); break;
        case 10: f(RadixTag<10>{}); break;
        default: f(RadixTag<12>{}); break;
    }
}

// The block's lines in shared memory, element i of line l at i SI + l SL: lines
// fastest (SI = LP, SL = 1) where neighbouring lines are neighbours in memory
// (y, x), elements fastest (SI = 1, SL = n) where a line is contiguous (z).
// Butterfly tasks t of a stage with nb butterflies a line run in the same order.
struct LineMap {
    int LP, si, sl;
    bool lines_first;
    __device__ __forceinline__ void task(int t, int nb, int& l, int& j) const
    {
        if (lines_first) {
            j = (int)((unsigned)t / (unsigned)LP);
            l = t - j * LP;
        } else {
            l = (int)((unsigned)t / (unsigned)nb);
            j = t - l * nb;
        }
    }
};

// First stage: radix r, inputs j + k n/r from load(l, index), outputs j r + k.
template <bool INV, typename R, typename C, typename Load>
__device__ __forceinline__ void fft_first(int n, int r, const LineMap& M, Load&& load, C* out)
{
    with_radix(r, [&](auto tag) {
        constexpr int N = decltype(tag)::value;
        const int nb = n / N;
        for (int t = threadIdx.x; t < M.LP * nb; t += FFT_THREADS) {
            int l, j;
            M.task(t, nb, l, j);
            C v[N];
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = load(l, j + k * nb);
            RDft<N, INV, R, C>::run(v);
            C* o = out + j * N * M.si + l * M.sl;
#pragma unroll
            for (int k = 0; k < N; ++k) o[k * M.si] = v[k];
        }
    });
}

// Middle stage: radix r after a first stage of radix ns.
template <bool INV, typename R, typename C>
__device__ __forceinline__ void fft_middle(int n, int ns, int r, const LineMap& M, const C* tw, const C* in, C* out)
{
    with_radix(r, [&](auto tag) {
        constexpr int N = decltype(tag)::value;
        const int nb = n / N, step = n / (ns * N);
        for (int t = threadIdx.x; t < M.LP * nb; t += FFT_THREADS) {
            int l, j;
            M.task(t, nb, l, j);
            const int q = (int)((unsigned)j / (unsigned)ns), m = j - q * ns;
            const C* p = in + j * M.si + l * M.sl;
            C v[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                v[k] = p[k * nb * M.si];
                if (k) {
                    const C w = tw[k * m * step];
                    v[k] = cmul(v[k], INV ? cconj(w) : w);
                }
            }
            RDft<N, INV, R, C>::run(v);
            C* o = out + (q * ns * N + m) * M.si + l * M.sl;
#pragma unroll
            for (int k = 0; k < N; ++k) o[k * ns * M.si] = v[k];
        }
    });
}

// Last stage: radix r after stages of product n/r; sink(l, j, nb, v): v[k] is
// element j + k nb of the transform.
template <bool INV, typename R, typename C, typename Sink>
__device__ __forceinline__ void fft_last(int n, int r, const LineMap& M, const C* tw, const C* in, Sink&& sink)
{
    with_radix(r, [&](auto tag) {
        constexpr int N = decltype(tag)::value;
        const int nb = n / N;
        for (int t = threadIdx.x; t < M.LP * nb; t += FFT_THREADS) {
            int l, j;
            M.task(t, nb, l, j);
            const C* p = in + j * M.si + l * M.sl;
            C v[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                v[k] = p[k * nb * M.si];
                if (k) {
                    const C w = tw[k * j];
                    v[k] = cmul(v[k], INV ? cconj(w) : w);
                }
            }
            RDft<N, INV, R, C>::run(v);
            sink(l, j, nb, v);
        }
    });
}

// Shared memory: twiddles [n] | two line buffers [LP n].
template <typename C>
struct FftSmem {
    C *tw, *a, *b;
    const C* g_tw;
    int n;
    C t0, t1;
    // The twiddles are on their way while the first stage loads and transforms.
    __device__ __forceinline__ FftSmem(unsigned char* raw, int n_, int LP, const C* __restrict__ g) : g_tw(g), n(n_)
    {
        tw = reinterpret_cast<C*>(raw);
        a = tw + n;
        b = a + LP * n;
        t0 = g[min((int)threadIdx.x, n - 1)];
        t1 = g[min((int)threadIdx.x + FFT_THREADS, n - 1)];
    }
    __device__ __forceinline__ void store() const
    {
        const int i = threadIdx.x;
        if (i < n) tw[i] = t0;
        if (i + FFT_THREADS < n) tw[i + FFT_THREADS] = t1;
        for (int k = i + 2 * FFT_THREADS; k < n; k += FFT_THREADS) tw[k] = g_tw[k];
    }
};

// Stages one and two of a forward or inverse transform: returns the buffer the
// last stage reads (after the barrier).  r2 == 1: no middle stage.
template <bool INV, typename R, typename C, typename Load>
__device__ __forceinline__ C* fft_to_last(int r1, int r2, const LineMap& M, const FftSmem<C>& S, Load&& load)
{
    fft_first<INV, R>(S.n, r1, M, load, S.a);
    S.store();
    __syncthreads();
    if (r2 == 1) return S.a;
    fft_middle<INV, R>(S.n, r1, r2, M, S.tw, S.a, S.b);
    __syncthreads();
    return S.b;
}

template <typename R>
__device__ __forceinline__ void regs_z_r2c_dev(const FFTZArgs<R>& A, int bx, int set)
{
    using C = typename CT<R>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = A.d.n, Kc = n / 2 + 1, LP = A.LP, nlines = A.nlines;
    const FftSmem<C> sm(smem_raw, n, LP, A.tw);
    C *const a = sm.a, *const b = sm.b;
    const C* tw = sm.tw;
    const LineMap M{LP, 1, n, false};
    const long long g0 = (long long)bx * 2 * LP;   // two real lines per complex one
    const unsigned long long* __restrict__ q = set ? A.qgrid2 : A.qgrid;
    C* __restrict__ cg = set ? A.cgrid2 : A.cgrid;
    auto value = [&](long long line, int z) {
        if (line >= nlines) return (R)0;
        const long long w = (long long)q[line * n + z];
        if (sizeof(R) == 4) return (R)(__ll2float_rn(w) * (float)GRID_ISCALE);
        return (R)((double)w * GRID_ISCALE);
    };
    C* in = fft_to_last<false, R>(A.d.r[0], A.d.r[1], M, sm, [&](int l, int z) {
        return C{value(g0 + 2 * l, z), value(g0 + 2 * l + 1, z)};
    });
    C* out = in == a ? b : a;
    fft_last<false, R>(n, A.d.r[2], M, tw, in, [&](int l, int j, int nb, auto& v) {
#pragma unroll
        for (int k = 0; k < (int)(sizeof(v) / sizeof(C)); ++k) out[l * n + j + k * nb] = v[k];
    });
    __syncthreads();
    for (int t = threadIdx.x; t < LP * Kc; t += FFT_THREADS) {
        const int l = (int)((unsigned)t / (unsigned)Kc), k = t - l * Kc;
        const C Z = out[l * n + k], Zc = cconj(out[l * n + (k == 0 ? 0 : n - k)]);
        const long long g = g0 + 2 * l;
        if (g < nlines) cg[g * Kc + k] = C{(R)0.5 * (Z.x + Zc.x), (R)0.5 * (Z.y + Zc.y)};
        if (g + 1 < nlines) cg[(g + 1) * Kc + k] = C{(R)0.5 * (Z.y - Zc.y), (R)-0.5 * (Z.x - Zc.x)};
    }
}

template <typename R>
__device__ __forceinline__ void regs_z_c2r_dev(const FFTZArgs<R>& A, int bx, int set)
{
    using C = typename CT<R>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = A.d.n, Kc = n / 2 + 1, LP = A.LP, nlines = A.nlines;
    const FftSmem<C> sm(smem_raw, n, LP, A.tw);
    const C* tw = sm.tw;
    const LineMap M{LP, 1, n, false};
    const long long g0 = (long long)bx * 2 * LP;
    const C* __restrict__ cg = set ? A.cgrid2 : A.cgrid;
    R* __restrict__ rg = set ? A.rgrid2 : A.rgrid;
    const C* in = fft_to_last<true, R>(A.d.r[0], A.d.r[1], M, sm, [&](int l, int k) {
        const long long g = g0 + 2 * l;
        const int kk = k < Kc ? k : n - k;
        C P = {0, 0}, Q = {0, 0};
        if (g < nlines) P = cg[g * Kc + kk];
        if (g + 1 < nlines) Q = cg[(g + 1) * Kc + kk];
        if (k >= Kc) {
            P = cconj(P);
            Q = cconj(Q);
        }
        // A real line's element 0 (and n/2) is real.  What the transforms before
        // left of an imaginary part is rounding, and through the packing it would
        // pass to the other line with opposite signs: an error of wavelength two
        // lines, which the force amplifies by K/2 (ordered water, FP32, relative
        // error of the forces: 216^3 4.1e-6 with it and 0.4e-6 without, the table-
        // driven passes 2.1e-6 with it; 144^3 and 192^3 2.4e-6 and 3.1e-6 -> 0.4e-6).
        if (k == 0 || 2 * k == n) P.y = Q.y = 0;
        return C{P.x - Q.y, P.y + Q.x};
    });
    fft_last<true, R>(n, A.d.r[2], M, tw, in, [&](int l, int j, int nb, auto& v) {
        const long long g = g0 + 2 * l;
#pragma unroll
        for (int k = 0; k < (int)(sizeof(v) / sizeof(C)); ++k) {
            if (g < nlines) rg[g * n + j + k * nb] = v[k].x;
            if (g + 1 < nlines) rg[(g + 1) * n + j + k * nb] = v[k].y;
        }
    });
}

template <typename R, bool INV>
__device__ __forceinline__ void regs_y_dev(const FFTYArgs<R>& A, int bx, int by, int set)
{
    using C = typename CT<R>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = A.d.n, Kc = A.Kc, LP = A.LP, kz0 = bx * LP;
    const FftSmem<C> sm(smem_raw, n, LP, A.tw);
    const C* tw = sm.tw;
    const LineMap M{LP, LP, 1, true};
    C* __restrict__ cg = (set ? A.cgrid2 : A.cgrid) + (long long)by * n * Kc + kz0;
    const int live = min(LP, Kc - kz0);
    const C* in = fft_to_last<INV, R>(A.d.r[0], A.d.r[1], M, sm, [&](int l, int y) {
        return l < live ? cg[(long long)y * Kc + l] : C{0, 0};
    });
    fft_last<INV, R>(n, A.d.r[2], M, tw, in, [&](int l, int j, int nb, auto& v) {
        if (l >= live) return;
#pragma unroll
        for (int k = 0; k < (int)(sizeof(v) / sizeof(C)); ++k) cg[(long long)(j + k * nb) * Kc + l] = v[k];
    });
}

// The influence function is laid out [ky][kx][kz] here: lanes run along kz.
template <typename R, bool ENERGY>
__device__ __forceinline__ void regs_x_conv_dev(const FFTXArgs<R>& A, int bx, int by, int set)
{
    using C = typename CT<R>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = A.d.n, Kc = A.Kc, K1 = A.K1, LP = A.LP, kz0 = bx * LP;
    const int y = by;
    const FftSmem<C> sm(smem_raw, n, LP, A.tw);
    C *const a = sm.a, *const b = sm.b;
    const C* tw = sm.tw;
    const LineMap M{LP, LP, 1, true};
    const long long stride = (long long)K1 * Kc;
    C* __restrict__ cg = (set ? A.cgrid2 : A.cgrid) + (long long)y * Kc + kz0;
    const R* __restrict__ fl = A.infl + (long long)y * n * Kc + kz0;
    const int live = min(LP, Kc - kz0);
    const int r1 = A.d.r[0], r2 = A.d.r[1], r3 = A.d.r[2];
    const C* in = fft_to_last<false, R>(r1, r2, M, sm, [&](int l, int x) {
        return l < live ? cg[x * stride + l] : C{0, 0};
    });
    C* turn = in == a ? b : a;
    double e_sum = 0, w6[6] = {0, 0, 0, 0, 0, 0};
    const bool energy = ENERGY && !A.cp.reference;
    if (!ENERGY) {
        fft_last<false, R>(n, r3, M, tw, in, [&](int l, int j, int nb, auto& v) {
            constexpr int N = (int)(sizeof(v) / sizeof(C));
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const R c = l < live ? fl[(long long)(j + k * nb) * Kc + l] : (R)0;
                v[k].x = mul_rn(v[k].x, c);
                v[k].y = mul_rn(v[k].y, c);
            }
            RDft<N, true, R, C>::run(v);   // first stage of the inverse with the radices reversed
            C* o = turn + j * N * M.si + l * M.sl;
#pragma unroll
            for (int k = 0; k < N; ++k) o[k * M.si] = v[k];
        });
        __syncthreads();
    } else {
        // With energies the transform goes through shared memory in between: the
        // FP64 sums unrolled over the radix cost 104 registers and instruction
        // fetches (216^3 121 us against 81).  A thread keeps one line.
        fft_last<false, R>(n, r3, M, tw, in, [&](int l, int j, int nb, auto& v) {
#pragma unroll
            for (int k = 0; k < (int)(sizeof(v) / sizeof(C)); ++k) turn[(j + k * nb) * LP + l] = v[k];
        });
        __syncthreads();
        const int per = FFT_THREADS / LP, i0 = threadIdx.x / LP, l = threadIdx.x - i0 * LP;
        if (i0 < per && l < live) {
            // em = c |S|^2 along a line (ky, kz fixed): the virial factor
            // 2 (1 + pa2 m2)/m2 splits into h = em/m2 and em, so five sums over kx
            // hold all six components (sum h mx^2 = sum em - (my^2 + mz^2) sum h)
            const double my = A.my[y], mz = A.mz[kz0 + l], myz2 = my * my + mz * mz;
            double s_e = 0, s_h = 0, s_ex = 0, s_hx = 0, s_em = 0;
            constexpr int U = 4;   // elements in flight
            for (int k0 = i0; k0 < n; k0 += U * per) {
                R c[U];
                double mx[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int kx = min(k0 + u * per, n - 1);
                    c[u] = fl[(long long)kx * Kc + l];
                    mx[u] = A.mx[kx];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int kx = k0 + u * per;
                    if (kx >= n) break;
                    C S = turn[kx * LP + l];
                    if (energy && c[u] != (R)0) {
                        const double em = (double)c[u] * ((double)S.x * S.x + (double)S.y * S.y);
                        const double m2 = fma(mx[u], mx[u], myz2);
                        double r = (double)rcp_ftz((float)m2);   // 1/m2: Newton's iteration r (2 - m2 r), twice
                        r = fma(r, fma(-m2, r, 1.0), r);
                        r = fma(r, fma(-m2, r, 1.0), r);
                        const double h = em * r;
                        s_e += em;
                        s_h += h;
                        s_ex = fma(em, mx[u], s_ex);
                        s_hx = fma(h, mx[u], s_hx);
                        s_em = fma(em, m2, s_em);
                    }
                    S.x *= c[u];
                    S.y *= c[u];
                    turn[kx * LP + l] = S;
                }
            }
            const int kz = kz0 + l;
            const double w = (kz == 0 || ((A.cp.K[2] & 1) == 0 && kz == A.cp.K[2] / 2)) ? 0.5 : 1.0;
            const double p2 = 2.0 * A.cp.pa2 * w, w2 = 2.0 * w;
            const double v0 = w2 * s_h + p2 * s_e;                                   // sum em vf
            const double vx = w2 * s_hx + p2 * s_ex;                                 // sum em vf mx
            const double vxx = w2 * (s_e - myz2 * s_h) + p2 * (s_em - myz2 * s_e);   // sum em vf mx^2
            e_sum = w * s_e;
            w6[0] = e_sum - vxx; w6[1] = -my * vx; w6[2] = -mz * vx;
            w6[3] = e_sum - my * my * v0; w6[4] = -my * mz * v0; w6[5] = e_sum - mz * mz * v0;
        }
        __syncthreads();
        C* first = turn == a ? b : a;
        fft_first<true, R>(n, r3, M, [&](int ll, int x) { return turn[x * LP + ll]; }, first);
        __syncthreads();
        turn = first;
    }
    C* back = turn;
    if (r2 != 1) {
        back = turn == a ? b : a;
        fft_middle<true, R>(n, r3, r2, M, tw, turn, back);
        __syncthreads();
    }
    fft_last<true, R>(n, r1, M, tw, back, [&](int l, int j, int nb, auto& v) {
        if (l >= live) return;
#pragma unroll
        for (int k = 0; k < (int)(sizeof(v) / sizeof(C)); ++k) cg[(j + k * nb) * stride + l] = v[k];
    });
    if (energy) {
        const double v[7] = {e_sum, w6[0], w6[1], w6[2], w6[3], w6[4], w6[5]};
        const int idx[7] = {MDF_E_EE_RECIP, ACC_VIR + 0, ACC_VIR + 1, ACC_VIR + 2, ACC_VIR + 3, ACC_VIR + 4,
                            ACC_VIR + 5};
        block_acc_fixed<7>(v, A.acc, idx, ENERGY_SCALE, A.st);
    }
}

// Radices of a length: two of {1..6, 8, 9, 10, 12} (r[1] = 1) or three, the
// largest as small as possible; r[0] = 0 when there are none.  r[0] is the
// first stage, r[2] the last.
inline void fft_radices(int n, int r[3])
{
    const int set[10] = {12, 10, 9, 8, 6, 5, 4, 3, 2, 1};
    r[0] = r[1] = r[2] = 0;
    int best = 99;
    for (int a : set)
        for (int b : set)
            if (a >= b && a * b == n && a < best) {
                best = a;
                r[0] = a;
                r[1] = 1;
                r[2] = b;
            }
    if (r[0]) return;
    for (int a : set)
        for (int b : set)
            for (int c : set)
                if (a >= b && b >= c && a * b * c == n && a < best) {
                    best = a;
                    r[0] = a;
                    r[1] = b;
                    r[2] = c;
                }
}

}  // namespace mdf
