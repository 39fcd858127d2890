/*
 * Spectral derivatives of one lattice line by folded circulant products.
 *
 * On a periodic line of n points the operators of the step along one axis, the laplacian part
 * -k^2 and the first derivative i k (Nyquist mode zeroed), are real circulant matrices: n-periodic
 * kernels t(d) with t(-d) = t(d) (laplacian) or t(-d) = -t(d) (derivative).  A thread applies
 * them to a real line it holds in registers:
 *
 *   the reflection j -> -j splits the line into an even and an odd half: the laplacian acts
 *     within each, the derivative from each to the other;
 *   the shift by n/2 splits the circulant of n points into a circulant of n/2 (p_j = f_j +
 *     f_{j+n/2}) and a skew-circulant, antiperiodic, of n/2 (m_j = f_j - f_{j+n/2}), within each
 *     half; recursively on p while n is even.
 *
 * For n = 32 the laplacian costs 174 multiply-adds and 164 additions of a real line, with
 * coefficients that are compile-time constants; the forward and inverse transforms it replaces
 * cost about 700 operations of a complex line each, with twiddle loads, exchanges between the
 * threads of a line and barriers.  Rounding is that of sums of n products with
 * sum_d |t(d)| = max k^2.
 */
#ifndef WTD_CIRC_CUH
#define WTD_CIRC_CUH

#include <cuda_runtime.h>
#include <type_traits>
#include "wtd_core.cuh"

namespace circ {

/* The coefficients are formed at compile time as unevaluated sums of two doubles (Dekker 1971, Numer.
 * Math. 18) and rounded once.  They are the same in every step, so their errors add up coherently
 * over a run: formed in plain doubles they made up nearly all of the operators' error (laplacian
 * of 12 points: 1.8e-16 of 1.9e-16 relative, rounded once 0.9e-16 of 1.4e-16). */
struct dd {
    double h, l;
};
constexpr dd fast_sum(double a, double b) { return dd{a + b, b - ((a + b) - a)}; }   /* |a| >= |b| */
constexpr dd two_sum(double a, double b)
{
    const double s = a + b, t = s - a;
    return dd{s, (a - (s - t)) + (b - t)};
}
constexpr dd two_prod(double a, double b)
{
    const double p = a * b, ca = 134217729.0 * a, cb = 134217729.0 * b;   /* 2^27 + 1 */
    const double ah = ca - (ca - a), al = a - ah, bh = cb - (cb - b), bl = b - bh;
    return dd{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr dd add(dd a, dd b)
{
    const dd s = two_sum(a.h, b.h), t = two_sum(a.l, b.l), u = fast_sum(s.h, s.l + t.h);
    return fast_sum(u.h, u.l + t.l);
}
constexpr dd neg(dd a) { return dd{-a.h, -a.l}; }
constexpr dd mul(dd a, dd b)
{
    const dd p = two_prod(a.h, b.h);
    return fast_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr dd scl(dd a, double b) { return mul(a, dd{b, 0.0}); }
constexpr dd quo(dd a, dd b)
{
    const double q = a.h / b.h;
    const dd r = add(a, neg(scl(b, q)));
    const double q2 = r.h / b.h;
    const dd r2 = add(r, neg(scl(b, q2)));
    return add(fast_sum(q, q2), dd{r2.h / b.h, 0.0});
}
constexpr dd PI2{3.14159265358979323846, 1.2246467991473531772e-16};   /* pi */

/* sin and cos of x in [0, pi/4] by their Taylor series, smallest terms first */
constexpr dd taylor(dd x, bool sine)
{
    dd term[16] = {}, t = sine ? x : dd{1.0, 0.0};
    const dd xx = neg(mul(x, x));
    for (int k = 0; k < 16; k++) {
        term[k] = t;
        t = quo(mul(t, xx), dd{sine ? (2.0 * k + 2.0) * (2.0 * k + 3.0) : (2.0 * k + 1.0) * (2.0 * k + 2.0), 0.0});
    }
    dd s{0.0, 0.0};
    for (int k = 15; k >= 0; k--) s = add(s, term[k]);
    return s;
}
/* pi m / n */
constexpr dd pi_frac(int m, int n) { return quo(scl(PI2, (double)m), dd{(double)n, 0.0}); }
/* sin(pi d / n), cos(pi d / n) for 0 <= d <= n, reduced exactly to [0, pi/4] */
constexpr dd sin_pi(int d, int n)
{
    return 2 * d > n ? sin_pi(n - d, n) : 4 * d > n ? taylor(pi_frac(n - 2 * d, 2 * n), false) : taylor(pi_frac(d, n), true);
}
constexpr dd cos_pi(int d, int n)
{
    return 2 * d > n ? neg(cos_pi(n - d, n)) : 4 * d > n ? taylor(pi_frac(n - 2 * d, 2 * n), true) : taylor(pi_frac(d, n), false);
}

enum { LAP = 0, DER = 1 };

/* kernel of the operator along axis AX on N points (N even) from the symbol that the transforms
 * apply, k_q = (2 pi / L) q and its square as doubles, Nyquist mode zeroed in the derivative:
 * laplacian t(d) = (1/N) sum_q -k_q^2 e^{2 pi i q d/N}, derivative t(d) = (1/N) sum_q i k_q
 * e^{2 pi i q d/N} */
template <int OP, int AX> constexpr double symbol(int q)
{
    const double k = 2.0 * PI2.h / (AX == 0 ? (double)(LX) : AX == 1 ? (double)(LY) : (double)(LZ)) * (double)q;
    return OP == LAP ? -(k * k) : -k;
}
/* kernel of the circulant block of n points inside a line of N: 2^-l sum_s t(d + s n), N = 2^l n,
 * from that of 2 n points */
template <int OP, int AX, int N, int n> struct Cyc {
    dd t[n];
    constexpr Cyc() : t()
    {
        if constexpr (n == N) {
            dd w[N] = {};   /* cos or sin (2 pi m / N) */
            for (int m = 0; 2 * m <= N; m++) w[m] = OP == LAP ? cos_pi(2 * m, N) : sin_pi(2 * m, N);
            for (int m = 1; 2 * m < N; m++) w[N - m] = OP == LAP ? w[m] : neg(w[m]);
            for (int d = 0; 2 * d <= N; d++) {
                dd s{0.0, 0.0};
                for (int q = N / 2 - 1; q > 0; q--) s = add(s, scl(w[q * d % N], 2.0 * symbol<OP, AX>(q)));
                if (OP == LAP) s = add(s, scl(w[N / 2 * d % N], symbol<OP, AX>(N / 2)));
                t[d] = quo(s, dd{(double)N, 0.0});
            }
            for (int d = 1; 2 * d < N; d++) t[N - d] = OP == LAP ? t[d] : neg(t[d]);
        } else {
            const Cyc<OP, AX, N, 2 * n> p;
            for (int d = 0; d < n; d++) t[d] = scl(add(p.t[d], p.t[d + n]), 0.5);
        }
    }
};
/* kernel of the skew block of n points (the m half of the circulant of 2 n points) */
template <int OP, int AX, int N, int n> struct Skw {
    dd t[n];
    constexpr Skw() : t()
    {
        const Cyc<OP, AX, N, 2 * n> p;
        for (int d = 0; d < n; d++) t[d] = scl(add(p.t[d], neg(p.t[d + n])), 0.5);
    }
};
/* either, at any d: periodic, or antiperiodic where skew */
template <int OP, int AX, int N, int n, bool SKEW> constexpr dd tk(int d)
{
    constexpr typename std::conditional<SKEW, Skw<OP, AX, N, n>, Cyc<OP, AX, N, n>>::type T;
    const int m = ((d % (2 * n)) + 2 * n) % (2 * n), r = m % n;
    return SKEW && m >= n ? neg(T.t[r]) : T.t[r];
}

/* even indices 0..ne-1 and odd indices 1..no of a block */
constexpr int n_even(int n, bool skew) { return skew ? (n + 1) / 2 : n / 2 + 1; }
constexpr int n_odd(int n, bool skew) { return skew ? n / 2 : (n - 1) / 2; }
/* k is its own mirror image in the even (odd) half */
constexpr bool self_even(int n, bool skew, int k) { return k == 0 || (!skew && 2 * k == n); }
constexpr bool self_odd(int n, bool skew, int k) { return skew && 2 * k == n; }

/* coefficient from even input k (EV) or odd input k to output row j */
template <int OP, int AX, int N, int n, bool SKEW, bool EV, int j, int k> struct Coef {
    static constexpr bool self = EV ? self_even(n, SKEW, k) : self_odd(n, SKEW, k);
    static constexpr dd a = tk<OP, AX, N, n, SKEW>(j - k), b = tk<OP, AX, N, n, SKEW>(j + k);
    static constexpr double value = self ? a.h : scl(add(a, EV ? b : neg(b)), 0.5).h;
};

template <int OP, int AX, int N, int n, bool SKEW, bool EV, int j, int k, int K1, typename R>
__device__ __forceinline__ R row(const R *in, R acc)
{
    if constexpr (k < K1) {
        constexpr double c = Coef<OP, AX, N, n, SKEW, EV, j, k>::value;
        return row<OP, AX, N, n, SKEW, EV, j, k + 1, K1>(in, c == 0.0 ? acc : acc + (R)c * in[k]);
    } else return acc;
}
/* rows j..J1-1: out[j] = sum_k coef(j, k) in[k], k = K0..K1-1 */
template <int OP, int AX, int N, int n, bool SKEW, bool EV, int j, int J1, int K0, int K1, typename R>
__device__ __forceinline__ void rows(const R *in, R *out)
{
    if constexpr (j < J1) {
        out[j] = row<OP, AX, N, n, SKEW, EV, j, K0, K1>(in, (R)0);
        rows<OP, AX, N, n, SKEW, EV, j + 1, J1, K0, K1>(in, out);
    }
}

/* the even (EV) or odd half of the circulant block of n points: in[k] are the folded inputs
 * f_k + f_{-k} (f_k where k is its own mirror image) or f_k - f_{-k}, out[j] the even or odd half
 * of the result, whose parity the derivative changes */
template <int OP, int AX, int N, int n, bool EV, typename R>
__device__ __forceinline__ void half(const R (&in)[n / 2 + 1], R (&out)[n / 2 + 1])
{
    constexpr bool OV = OP == LAP ? EV : !EV;
    if constexpr (n % 2 == 0 && n >= 4) {
        /* circulant (p) and skew (m) blocks of h = n/2 points: the half-shift folds the half onto
         * itself, k -> h - k */
        constexpr int h = n / 2;
        R pi[h / 2 + 1], po[h / 2 + 1], mi[h / 2 + 1], mo[h / 2 + 1];
        if constexpr (EV) {
#pragma unroll
            for (int k = 0; k < n_even(h, false); k++) pi[k] = 2 * k == h ? in[k] : in[k] + in[h - k];
#pragma unroll
            for (int k = 0; k < n_even(h, true); k++) mi[k] = in[k] - in[h - k];
        } else {
#pragma unroll
            for (int k = 1; k <= n_odd(h, false); k++) pi[k] = in[k] - in[h - k];
#pragma unroll
            for (int k = 1; k <= n_odd(h, true); k++) mi[k] = 2 * k == h ? in[k] : in[k] + in[h - k];
        }
        rows<OP, AX, N, h, true, EV, OV ? 0 : 1, OV ? n_even(h, true) : n_odd(h, true) + 1, EV ? 0 : 1,
             EV ? n_even(h, true) : n_odd(h, true) + 1>(mi, mo);
        half<OP, AX, N, h, EV>(pi, po);
        if constexpr (OV) {
#pragma unroll
            for (int j = 0; 2 * j <= h; j++) {
                if (2 * j == h) out[j] = po[j];
                else { out[j] = po[j] + mo[j]; out[h - j] = po[j] - mo[j]; }
            }
        } else {
#pragma unroll
            for (int j = 1; 2 * j <= h; j++) {
                if (2 * j == h) out[j] = mo[j];
                else { out[j] = po[j] + mo[j]; out[h - j] = mo[j] - po[j]; }
            }
        }
    } else {
        rows<OP, AX, N, n, false, EV, OV ? 0 : 1, OV ? n_even(n, false) : n_odd(n, false) + 1, EV ? 0 : 1,
             EV ? n_even(n, false) : n_odd(n, false) + 1>(in, out);
    }
}

/* sources of a line: in registers, or in memory at a run-time step.  A memory line is read again for
 * the second half, through a step made opaque so that neither the values nor their addresses are
 * kept in registers in between (at 64 points in FP64 that is the difference to spilling) */
template <typename R, int N> struct RegLine {
    const R (&v)[N];
    __device__ __forceinline__ R operator()(int k) const { return v[k]; }
    __device__ __forceinline__ void again() {}
};
template <typename R> struct MemLine {
    const R *p;
    int st;
    __device__ __forceinline__ R operator()(int k) const { return p[k * st]; }
    __device__ __forceinline__ void again() { asm volatile("" : "+r"(st) : : "memory"); }
};

/* y = (laplacian part or derivative along axis AX) of the line f(0..N-1), N even */
template <int OP, int AX, int N, class F, typename R>
__device__ __forceinline__ void line_from(F &f, R (&y)[N])
{
    constexpr int H = N / 2;
    R g[H + 1], h[H + 1];
    {
        R e[H + 1];
#pragma unroll
        for (int k = 0; k <= H; k++) e[k] = (k == 0 || k == H) ? f(k) : f(k) + f(N - k);
        if constexpr (OP == LAP) half<OP, AX, N, N, true>(e, g);
        else half<OP, AX, N, N, true>(e, h);
    }
    f.again();
    {
        R o[H + 1];
#pragma unroll
        for (int k = 1; k < H; k++) o[k] = f(k) - f(N - k);
        if constexpr (OP == LAP) half<OP, AX, N, N, false>(o, h);
        else half<OP, AX, N, N, false>(o, g);
    }
    y[0] = g[0];
    y[H] = g[H];
#pragma unroll
    for (int j = 1; j < H; j++) { y[j] = g[j] + h[j]; y[N - j] = g[j] - h[j]; }
}
template <int OP, int AX, int N, typename R>
__device__ __forceinline__ void line_op(const R (&f)[N], R (&y)[N])
{
    RegLine<R, N> r{f};
    line_from<OP, AX, N>(r, y);
}

} // namespace circ

/* ---------------------------------------------------------------------------------------
 * Lines of a lattice field in shared memory.  A field is complex, natural order, rows of the
 * fastest axis padded to an odd length, so that the lines of every axis fall on distinct banks.
 * A line is one real component (re or im) of the points along one axis: the lines of all axes
 * are numbered axis by axis, the re and im lines of the same points on adjacent threads.
 * -------------------------------------------------------------------------------------*/
template <class G> struct CircGeo {
    static constexpr int dims = G::dims, ntot = G::ntot, nfast = G::nfast, rows = G::rows;
    static constexpr int n(int a) { return G::n(a); }
    static constexpr int nmax = (n(0) > n(1) ? n(0) : n(1)) > n(2) ? (n(0) > n(1) ? n(0) : n(1)) : n(2);
    /* up to 64 points a line stays in one thread's registers (FusedCfg and AdjCfg set lower limits
     * for their kernels).  A 1D lattice has two lines only, so beyond 32 points the transforms,
     * which share a line among threads, are the better form */
    static constexpr bool fits = nmax <= 64 && (dims > 1 || nmax <= 32);
    static constexpr int pitch = nfast | 1, padded = rows * pitch;
    __host__ __device__ static constexpr int off(int i) { return (i / nfast) * pitch + i % nfast; }
    __host__ __device__ static constexpr int nlines(int a) { return a < dims ? 2 * ntot / n(a) : 0; }
    __host__ __device__ static constexpr int first(int a) { return (a > 0 ? nlines(0) : 0) + (a > 1 ? nlines(1) : 0); }
    static constexpr int total = nlines(0) + nlines(1) + nlines(2);
    /* all axes alike: one instance of the line operator serves them */
    static constexpr bool uniform = (dims < 2 || (n(0) == n(1) && (double)(DX) == (double)(DY))) &&
                                    (dims < 3 || (n(0) == n(2) && (double)(DX) == (double)(DZ)));
};

template <class CG> struct CircLine {
    bool on;
    int ax, c;       /* axis, 0 re / 1 im */
    int base, st;    /* real index of the first point in the padded field, and the step */
    int pb, ps;      /* natural index of the first point, and the step */
    __device__ __forceinline__ CircLine(int l)
    {
        on = l < CG::total;
        if (!on) l = l & 1;
        ax = (CG::dims > 2 && l >= CG::first(2)) ? 2 : (CG::dims > 1 && l >= CG::first(1)) ? 1 : 0;
        l -= ax == 2 ? CG::first(2) : ax == 1 ? CG::first(1) : 0;
        c = l & 1;
        const int o = l >> 1;
        int e;          /* padded element of the first point */
        if (CG::dims == 1) { e = 0; st = 1; pb = 0; ps = 1; }
        else if (CG::dims == 2) {
            if (ax == 0) { e = o; st = CG::pitch; pb = o; ps = CG::n(1); }
            else { e = o * CG::pitch; st = 1; pb = o * CG::n(1); ps = 1; }
        } else if (ax == 0) { e = (o / CG::n(2)) * CG::pitch + o % CG::n(2); st = CG::n(1) * CG::pitch; pb = o; ps = CG::n(1) * CG::n(2); }
        else if (ax == 1) {
            const int x = o / CG::n(2), z = o - x * CG::n(2);
            e = x * CG::n(1) * CG::pitch + z; st = CG::pitch; pb = x * CG::n(1) * CG::n(2) + z; ps = CG::n(2);
        } else { e = o * CG::pitch; st = 1; pb = o * CG::n(2); ps = 1; }
        base = 2 * e + c;
        st *= 2;
        /* opaque, so that the addresses of a line's points are formed where they are used: they do
         * not change from state to state and would otherwise be kept across the state loop, in
         * local memory (600 bytes a thread at 48 points in FP64) */
        asm volatile("" : "+r"(base), "+r"(st), "+r"(pb), "+r"(ps));
    }
};

template <int A> struct CircAxis { static constexpr int value = A; };
/* f(axis constant) for a runtime axis; uniform lattices take axis 0's instance */
template <class CG, class F> __device__ __forceinline__ void circ_axis(int ax, F f)
{
    if constexpr (CG::uniform) f(CircAxis<0>());
    else {
        if (ax == 0) f(CircAxis<0>());
        else if (CG::dims == 2 || ax == 1) { if constexpr (CG::dims >= 2) f(CircAxis<1>()); }
        else { if constexpr (CG::dims >= 3) f(CircAxis<2>()); }
    }
}

/* the block's lines of a round write v into dst one axis after the other: axis 0 assigns (or adds
 * where ADD), the others add; every point has one line per axis, so no two threads of a phase
 * share a word.  Ends with a barrier. */
template <class CG, bool ADD, typename R>
__device__ __forceinline__ void circ_store(R *dst, const CircLine<CG> &L, const R (&v)[CG::nmax], int r0)
{
#pragma unroll
    for (int a = 0; a < CG::dims; a++) {
        if (r0 >= CG::first(a) + CG::nlines(a) || r0 + (int)blockDim.x <= CG::first(a)) continue;
        if (L.on && L.ax == a) {
            int st = L.st;
            asm volatile("" : "+r"(st));   /* addresses formed here, not kept from the loads */
#pragma unroll
            for (int j = 0; j < CG::nmax; j++)
                if (j < CG::n(a)) {
                    R &w = dst[L.base + j * st];
                    w = (a > 0 || ADD) ? w + v[j] : v[j];
                }
        }
        __syncthreads();
    }
}

/* dst = laplacian of src (padded complex fields in shared memory).  INPLACE: dst is src, and all
 * lines are held by the block at once (CG::total threads) */
template <class CG, bool INPLACE, typename C>
__device__ __forceinline__ void circ_lap(const C *src, C *dst)
{
    typedef decltype(src[0].x) RC;
    typedef typename std::remove_const<RC>::type R;
    const R *s = (const R *)src;
#pragma unroll 1
    for (int r0 = 0; r0 < CG::total; r0 += blockDim.x) {
        const CircLine<CG> L(r0 + threadIdx.x);
        R v[CG::nmax];
        if (L.on)
            circ_axis<CG>(L.ax, [&](auto A) {
                constexpr int AX = decltype(A)::value, n = CG::n(AX);
                R l[n];
                circ::MemLine<R> f{s + L.base, L.st};
                circ::line_from<circ::LAP, AX, n>(f, l);
#pragma unroll
                for (int j = 0; j < n; j++) v[j] = l[j];
            });
        if (INPLACE) __syncthreads();
        circ_store<CG, false>((R *)dst, L, v, r0);
    }
}

/* dst (padded, shared memory) = laplacian of the component y stored in natural order (global
 * memory; a 3D lattice's lines are read in whole segments of the fastest axis or from L1) */
template <class CG, typename C>
__device__ __forceinline__ void circ_lap_from(const C *y, C *dst)
{
    typedef typename std::remove_const<decltype(y[0].x)>::type RC;
    typedef typename std::remove_const<RC>::type R;
#pragma unroll 1
    for (int r0 = 0; r0 < CG::total; r0 += blockDim.x) {
        const CircLine<CG> L(r0 + threadIdx.x);
        R v[CG::nmax];
        if (L.on)
            circ_axis<CG>(L.ax, [&](auto A) {
                constexpr int AX = decltype(A)::value, n = CG::n(AX);
                R l[n];
                circ::MemLine<R> f{(const R *)y + 2 * L.pb + L.c, 2 * L.ps};
                circ::line_from<circ::LAP, AX, n>(f, l);
#pragma unroll
                for (int j = 0; j < n; j++) v[j] = l[j];
            });
        circ_store<CG, false>((R *)dst, L, v, r0);
    }
}

#endif
