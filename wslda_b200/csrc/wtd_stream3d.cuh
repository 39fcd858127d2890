/*
 * The stream path: one TD half step on 3D lattices whose state does not fit one CTA (32^3,
 * 48^3, ...), whose axes have at most 64 points and whose plane and column blocks fit shared memory
 * (StreamFit in wtd_api.cuh: all such lattices with constant mass or in the FP32-mixed forms; with
 * variable mass in FP64 a (y, z) plane of up to 64 x 62 points, 64 x 64 is 512 bytes too large).
 *
 * Against the staged path in FP64, ms per step: 64^3 constant mass 200 states 17.0 / 20.6 (lines of 64
 * points spill in the density and x kernels, 4.7, 1.0 and 0.4 KB a thread, and still win); 50x54x64
 * 300 states 15.5 / 22.1, 10 states 1.02 / 2.71; 48^3 601 states 13.5 / 25.1; 32^3 variable mass 1500
 * states 14.0 / 29.3.  64^3 variable mass in FP64 stays on the staged path (200 states: 42.5).
 *
 * Every derivative is a folded circulant product of one real lattice line in one thread's
 * registers (wtd_circ.cuh), so a half step is a chain of plain streaming kernels:
 *
 *   k3s_plane_h     one CTA per (component, x-plane, chunk of states): the (y, z) part of the
 *                   kinetic and current terms of H psi (pca_kernels.cu:233-391) into h, unscaled;
 *   k3s_x_h         one CTA per (block of (y, z) columns, chunk of states): h += the x-line part
 *                   and the local terms; partial sums of <psi|H|psi>;
 *   k3s_abm         elementwise: f = h - <H> psi, the ABM predictor or corrector
 *                   (tdwslda_ode_integrator.h:26-220), partial sums of the norm;
 *   k3s_dens_*      densities of the updated states (pca_dens.cu:13-338): nu and rho per point,
 *                   and on gradient half steps tau and j along the plane's and the x lines.
 *
 * The updated states are stored before their norm is known.  What is formed from them next is
 * linear in the state (h) or quadratic (<H>, densities), so those kernels work on the stored values
 * and the state's scale 1/norm (k3s_sum) is taken in FP64 where the result is next used or summed.
 * The last half step of a call leaves normalised states, whose densities are summed from what is
 * stored: in FP64 scaled in place (k3s_rescale), in the complex64 forms stored after a pass for the
 * norm (k3s_abm, PASS 4 and 5).  Precision forms as in the fused pass: TY storage of the states, TH of the ABM history, TC of the derivatives;
 * local terms, ABM sums, norms, <H> and density sums are FP64.
 */
#ifndef WTD_STREAM3D_CUH
#define WTD_STREAM3D_CUH

#include "wtd_circ.cuh"
#include "wtd_step.cuh"

#if CODEDIM == 3
#define WTD_S3_NYZ ((NY) * (NZ))

/* the lattice geometry of the stream kernels */
struct S3 {
    static constexpr int N = (NX) * (NY) * (NZ), NYZ = WTD_S3_NYZ;
    static constexpr bool ok = NX <= 64 && NY <= 64 && NZ <= 64;
    /* threads of one plane: one per (line, re/im) of the wider set of lines */
    static constexpr int LT = (2 * (NY > NZ ? NY : NZ) + 31) / 32 * 32;
    /* plane rows of NZ + 1 elements (odd): lines along either axis fall on distinct banks */
    static constexpr int PITCH = NZ + 1, PL = NY * PITCH;
    /* (y, z) columns per CTA of the x kernels; both extents are even, so 4 always divides */
    static constexpr int QB = NYZ % 16 == 0 ? 16 : NYZ % 8 == 0 ? 8 : 4;
    static constexpr int NQB = NYZ / QB;
    static constexpr int XL = 2 * QB;                       /* threads of one (state, component) */
    static constexpr int XS = 64 / XL;                      /* states in flight (whole warps for any QB) */
    static constexpr unsigned XM = 2 * XL >= 32 ? 0xffffffffu : (1u << (2 * XL)) - 1u;   /* lanes of k3s_dens_x */
    /* elements per CTA of k3s_abm along one component; 2 ACH CTAs a state */
    static constexpr int AT = 256, AE = 4, ACH = (N + AT * AE - 1) / (AT * AE);
    /* grid of 2 ACH CTAs for each of S states: the states over y and z, whose extents stop at 65535
     * (all in x, with a division per CTA, took 1% of a step in the all-FP32 form) */
    static dim3 states_grid(int S)
    {
        const unsigned z = ((unsigned)S + 65534u) / 65535u;
        return dim3(2 * ACH, ((unsigned)S + z - 1) / z, z);
    }
};

/* ---- shared memory of the plane kernel: coefficient planes (variable mass), then per state in
 * flight the psi plane and the K plane */
template <typename TC, bool VAR> struct S3PlaneSmem {
    typedef typename cplx<TC>::t C;
    static constexpr size_t cfp = VAR ? ((size_t)3 * S3::PL * sizeof(TC) + 15) / 16 * 16 : 0;
    static constexpr size_t state = 2 * (size_t)S3::PL * sizeof(C);
    static constexpr bool ok = cfp + state <= WTD_SMEM_MAX;
    /* two states in flight share the coefficient planes where two such CTAs fit an SM */
    static constexpr int NS = VAR && 2 * (cfp + 2 * state + 1024) <= 233472 ? 2 : 1;
    static constexpr size_t bytes = cfp + NS * state;
};

template <typename TY, typename TC, bool VAR>
__global__ void __launch_bounds__(S3::LT * S3PlaneSmem<TC, VAR>::NS)
k3s_plane_h(const TY *__restrict__ Y, typename cplx<TC>::t *__restrict__ K, const double *__restrict__ cf, int S)
{
    typedef typename cplx<TC>::t C;
    typedef S3PlaneSmem<TC, VAR> SM;
    constexpr int N = S3::N, NYZ = S3::NYZ, LT = S3::LT, PITCH = S3::PITCH, PL = S3::PL, NS = SM::NS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TC *al = (TC *)smem_raw, *Ay = al + PL, *Az = Ay + PL;
    const int slot = threadIdx.x / LT, t = threadIdx.x - slot * LT;
    C *P = (C *)(smem_raw + SM::cfp + (size_t)slot * SM::state);
    TC *Pr = (TC *)P, *Kr = Pr + 2 * PL;
    const int pr = (int)(blockIdx.x % (2 * NX)), chunk = (int)(blockIdx.x / (2 * NX)), nch = (int)(gridDim.x / (2 * NX));
    const int comp = pr / NX, x = pr - comp * NX;
    if (VAR) {
        const double *a = cf + (size_t)(CF_ALA + comp) * N + (size_t)x * NYZ;
        const double *b = cf + (size_t)(comp ? CF_ABY : CF_AAY) * N + (size_t)x * NYZ;
        const double *d = cf + (size_t)(comp ? CF_ABZ : CF_AAZ) * N + (size_t)x * NYZ;
        for (int i = threadIdx.x; i < NYZ; i += LT * NS) {
            const int o = (i / NZ) * PITCH + i % NZ;
            al[o] = (TC)a[i]; Ay[o] = (TC)b[i]; Az[o] = (TC)d[i];
        }
    }
    const TC s4 = comp ? (TC)0.25 : (TC)-0.25;   /* -1/4 with the component's sign */
    const int line = t >> 1, c = t & 1;
    const TC sd = c ? (TC)1 : (TC)-1;            /* (-i A) d psi: re gains A d im, im gains -A d re */
    for (int n0 = NS * chunk; n0 < S; n0 += NS * nch) {
        const int n = n0 + slot;
        const bool act = n < S;
        const size_t base = ((size_t)comp * S + n) * N + (size_t)x * NYZ;
        /* the plane of the CTA's next state on its way to L2 while this one is worked on */
        if (t == 0 && n + NS * nch < S) prefetch_l2(Y + base + (size_t)NS * nch * N, NYZ * sizeof(TY));
        __syncthreads();
        if (act) {
#pragma unroll 8
            for (int i = t; i < NYZ; i += LT) {
                const TY a = Y[base + i];
                C z; z.x = a.x; z.y = a.y;
                P[(i / NZ) * PITCH + i % NZ] = z;
            }
        }
        __syncthreads();
        /* z lines: thread (row, re/im) */
        {
            const bool on = act && line < NY;
            const int o = 2 * line * PITCH;
            TC f[NZ];
            if (on) {
#pragma unroll
                for (int j = 0; j < NZ; j++) f[j] = Pr[o + 2 * j + c];
                if (VAR) {
                    TC d[NZ];
                    circ::line_op<circ::DER, 2, NZ>(f, d);
#pragma unroll
                    for (int j = 0; j < NZ; j++) Kr[o + 2 * j + 1 - c] = sd * Az[line * PITCH + j] * d[j];
                }
            }
            if (VAR) __syncthreads();
            if (on) {
                TC l[NZ];
                circ::line_op<circ::LAP, 2, NZ>(f, l);
                if (VAR) {
#pragma unroll
                    for (int j = 0; j < NZ; j++) {
                        const TC a = al[line * PITCH + j];
                        Kr[o + 2 * j + c] += s4 * a * l[j];
                        f[j] *= a;
                    }
                    circ::line_op<circ::LAP, 2, NZ>(f, l);
#pragma unroll
                    for (int j = 0; j < NZ; j++) Kr[o + 2 * j + c] += s4 * l[j];
                } else {
#pragma unroll
                    for (int j = 0; j < NZ; j++) Kr[o + 2 * j + c] = l[j];
                }
            }
        }
        __syncthreads();
        /* y lines: thread (column, re/im); the finished plane goes out */
        {
            const bool on = act && line < NZ;
            const int o = 2 * line;
            TC f[NY];
            if (on) {
#pragma unroll
                for (int j = 0; j < NY; j++) f[j] = Pr[o + 2 * j * PITCH + c];
                if (VAR) {
                    TC d[NY];
                    circ::line_op<circ::DER, 1, NY>(f, d);
#pragma unroll
                    for (int j = 0; j < NY; j++) Kr[o + 2 * j * PITCH + 1 - c] += sd * Ay[j * PITCH + line] * d[j];
                }
            }
            if (VAR) __syncthreads();
            if (on) {
                TC *out = (TC *)K + 2 * base + o + c;
                TC l[NY];
                circ::line_op<circ::LAP, 1, NY>(f, l);
                if (VAR) {
#pragma unroll
                    for (int j = 0; j < NY; j++) {
                        const TC a = al[j * PITCH + line];
                        Kr[o + 2 * j * PITCH + c] += s4 * a * l[j];
                        f[j] *= a;
                    }
                    circ::line_op<circ::LAP, 1, NY>(f, l);
#pragma unroll
                    for (int j = 0; j < NY; j++) out[2 * j * NZ] = Kr[o + 2 * j * PITCH + c] + s4 * l[j];
                } else {
#pragma unroll
                    for (int j = 0; j < NY; j++) out[2 * j * NZ] = Kr[o + 2 * j * PITCH + c] + l[j];
                }
            }
        }
    }
}

/* ---- shared memory of the x kernel: FP64 slabs of the local-term coefficients at the CTA's
 * columns (V + lap alpha/4 of both spins, Delta and, with variable mass, -div A/2 of both), the
 * compute-precision slabs (alpha and A_x of both, or the kinetic coefficient), then per state in
 * flight the state's values and, with variable mass, the H of both components */
template <typename TC, bool VAR> struct S3XSmem {
    typedef typename cplx<TC>::t C;
    static constexpr int SL = NX * S3::QB;
    static constexpr int NLOC = VAR ? 6 : 4, NTC = VAR ? 4 : 2;
    static constexpr size_t slabs = ((size_t)NLOC * SL * sizeof(double) + (size_t)NTC * SL * sizeof(TC) + 15) / 16 * 16;
    static constexpr size_t state = (VAR ? 4 : 2) * (size_t)SL * sizeof(C);
    static constexpr bool ok = slabs + S3::XS * state <= WTD_SMEM_MAX;
    /* states in flight: enough for whole warps, more where two CTAs still fit an SM */
    static constexpr int N0 = S3::XS > 1 ? S3::XS : 1;
    static constexpr int NS = 2 * (slabs + 2 * N0 * state + 1024) <= 233472 ? 2 * N0 : N0;
    static constexpr size_t bytes = slabs + NS * state;
};

/* barrier of the T threads that work on one state (whole warps where T is, else within the warp) */
template <int T> __device__ __forceinline__ void state_sync(int slot)
{
    if constexpr (T >= 64) asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(T) : "memory");
    else __syncwarp();
}

template <typename TY, typename TC, bool VAR>
__global__ void __launch_bounds__(2 * S3::XL * S3XSmem<TC, VAR>::NS)
k3s_x_h(const TY *__restrict__ Y, typename cplx<TC>::t *K, const double *__restrict__ cf, double *__restrict__ epart, int S)
{
    typedef typename cplx<TC>::t C;
    typedef S3XSmem<TC, VAR> SM;
    constexpr int N = S3::N, NYZ = S3::NYZ, QB = S3::QB, XL = S3::XL, NS = SM::NS, SL = SM::SL, T = 2 * XL * NS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *Wl = (double *)smem_raw;                       /* [NLOC][x][q]: W_a, W_b, Re D, Im D, cj_a, cj_b */
    TC *Tl = (TC *)(Wl + SM::NLOC * SL);                   /* [NTC][x][q]: alpha_a, alpha_b, Ax_a, Ax_b | aa, ab */
    const int qb = (int)(blockIdx.x % S3::NQB), chunk = (int)(blockIdx.x / S3::NQB), nch = (int)(gridDim.x / S3::NQB);
    const int q0 = qb * QB;
    for (int i = threadIdx.x; i < SL; i += T) {
        const size_t p = (size_t)(i / QB) * NYZ + q0 + i % QB;
        Wl[i] = VAR ? cf[CF_VA * (size_t)N + p] + cf[CF_NA * (size_t)N + p] : cf[CF_VA * (size_t)N + p];
        Wl[SL + i] = VAR ? cf[CF_VB * (size_t)N + p] + cf[CF_NB * (size_t)N + p] : cf[CF_VB * (size_t)N + p];
        Wl[2 * SL + i] = cf[CF_DRE * (size_t)N + p];
        Wl[3 * SL + i] = cf[CF_DIM * (size_t)N + p];
        if (VAR) {
            Wl[4 * SL + i] = cf[CF_CJA * (size_t)N + p];
            Wl[5 * SL + i] = cf[CF_CJB * (size_t)N + p];
            Tl[i] = (TC)cf[CF_ALA * (size_t)N + p];
            Tl[SL + i] = (TC)cf[CF_ALB * (size_t)N + p];
            Tl[2 * SL + i] = (TC)cf[CF_AAX * (size_t)N + p];
            Tl[3 * SL + i] = (TC)cf[CF_ABX * (size_t)N + p];
        } else {
            Tl[i] = (TC)cf[CF_AA * (size_t)N + p];
            Tl[SL + i] = (TC)cf[CF_AB * (size_t)N + p];
        }
    }
    const int g = threadIdx.x / XL, lane = threadIdx.x - g * XL;
    const int slot = g >> 1, comp = g & 1, q = lane >> 1, c = lane & 1;
    C *Yo = (C *)(smem_raw + SM::slabs + (size_t)slot * SM::state) + comp * SL;      /* own component */
    C *Yx = (C *)(smem_raw + SM::slabs + (size_t)slot * SM::state) + (1 - comp) * SL; /* the other */
    TC *Hr = (TC *)((C *)(smem_raw + SM::slabs + (size_t)slot * SM::state) + 2 * SL + comp * SL);
    const double *W = Wl + comp * SL, *Dr = Wl + 2 * SL, *Di = Wl + 3 * SL, *cj = Wl + (4 + comp) * SL;
    const TC *al = Tl + comp * SL, *Ax = Tl + (2 + comp) * SL;
    const TC sgn = comp ? (TC)-1 : (TC)1, s4 = comp ? (TC)0.25 : (TC)-0.25, sd = c ? (TC)1 : (TC)-1;
    const double sp = comp ? -1.0 : 1.0;
    /* D v (u rows) and D* u (v rows): re = Dr o.x -+ Di o.y, im = Dr o.y +- Di o.x; the current
     * term +- i cj psi adds -+ cj im to re and +- cj re to im for u, and both signs equal for v */
    const double sdi = (c ? 1.0 : -1.0) * sp, scj = c ? 1.0 : -1.0;
    __syncthreads();
    for (int n0 = NS * chunk; n0 < S; n0 += NS * nch) {
        const int n = n0 + slot;
        const bool act = n < S;
        const size_t base = ((size_t)comp * S + n) * N + q0 + q;     /* complex element (x = 0) */
        TC f[NX], l[NX];
        /* row segments of the CTA's next state (psi and K) on their way to L2 */
        if (n + NS * nch < S) {
            const size_t nb = ((size_t)comp * S + n + NS * nch) * N + q0;
            for (int r = lane; r < 2 * NX; r += XL) {
                const size_t o = nb + (size_t)(r >> 1) * NYZ;
                if (r & 1) prefetch_l2(K + o, QB * sizeof(C));
                else prefetch_l2(Y + o, QB * sizeof(TY));
            }
        }
        if (act) {
            const TC *yr = (const TC *)Y + 2 * base + c;
#pragma unroll
            for (int x = 0; x < NX; x++) f[x] = yr[(size_t)2 * x * NYZ];
#pragma unroll
            for (int x = 0; x < NX; x++) ((TC *)Yo)[2 * (x * QB + q) + c] = f[x];
            if (VAR) {
                circ::line_op<circ::DER, 0, NX>(f, l);
#pragma unroll
                for (int x = 0; x < NX; x++) Hr[2 * (x * QB + q) + 1 - c] = sd * Ax[x * QB + q] * l[x];
            }
        }
        state_sync<2 * XL>(slot);
        double e = 0.0;
        if (act) {
            circ::line_op<circ::LAP, 0, NX>(f, l);
            if (VAR) {
#pragma unroll
                for (int x = 0; x < NX; x++) {
                    const TC a = al[x * QB + q];
                    Hr[2 * (x * QB + q) + c] += s4 * a * l[x];
                    f[x] *= a;
                }
                circ::line_op<circ::LAP, 0, NX>(f, l);
            }
            TC *kr = (TC *)K + 2 * base + c;
#pragma unroll
            for (int x = 0; x < NX; x++) {
                const int i = x * QB + q;
                const C ys = Yo[i], yo = Yx[i];
                const double own = c ? (double)ys.y : (double)ys.x, par = c ? (double)ys.x : (double)ys.y;
                const double oc = c ? (double)yo.y : (double)yo.x, op = c ? (double)yo.x : (double)yo.y;
                const TC k0 = kr[(size_t)2 * x * NYZ];
                const TC kin = VAR ? k0 + Hr[2 * i + c] + s4 * l[x] : sgn * al[i] * (k0 + l[x]);
                double h = sp * W[i] * own + (Dr[i] * oc + sdi * Di[i] * op);
                if (VAR) h += scj * cj[i] * par;
                h += (double)kin;
                const TC hs = (TC)h;
                kr[(size_t)2 * x * NYZ] = hs;
                e += own * (double)hs;
            }
        }
#pragma unroll
        for (int o = XL / 2; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o, XL < 32 ? XL : 32);
        if (act && lane == 0) epart[(size_t)n * (2 * S3::NQB) + 2 * qb + comp] = e;
        state_sync<2 * XL>(slot);
    }
}

/* DV sum of the np partial sums of state n, one warp per state, fixed order.  norm: out[n] = 1 / sqrt of
 * it, the state's scale; else out[n] = it times the square of the scale sc[n] (the partial sums of
 * <H> are of the stored states) */
__global__ void __launch_bounds__(128) k3s_sum(const double *part, int np, int S, double *out, int norm, const double *sc)
{
    const int n = (int)(blockIdx.x * 4 + threadIdx.x / 32), lane = threadIdx.x & 31;
    if (n >= S) return;
    double s = 0.0;
    for (int k = lane; k < np; k += 32) s += part[(size_t)n * np + k];
    s = warp_sum(s) * WTD_DV;
    if (lane == 0) out[n] = norm ? 1.0 / sqrt(s) : s * (sc[n] * sc[n]);
}

/* the ABM update of one chunk of one component of one state, y and h times the state's scale.  PASS 0:
 * f_k = h - E y (or read from ring slot NH-1), predictor into y, partial corrector P; 1: corrector
 * into y; 2: norm only; 3: f_k only; 4: norm of the corrector, nothing stored; 5: corrector times the
 * scale scn of its norm into y.  4 and 5 end a call in the complex64 forms: the normalised value is
 * rounded once.  Scaling the rounded corrector in place would leave it as it is where the scale is
 * closer to 1 than half a unit of FP32, and with it a norm off by up to 3e-8 (48^3, 256 states, 20
 * steps: density error 4.9e-8 against 3.3e-8) */
template <typename TY, typename TH, typename TC, int NH, int PASS>
__global__ void __launch_bounds__(S3::AT) k3s_abm(StepArgs a, const typename cplx<TC>::t *__restrict__ H,
                                                  const double *__restrict__ sc, const double *__restrict__ scn,
                                                  double *__restrict__ npart)
{
    constexpr bool CORR = PASS == 1 || PASS == 4 || PASS == 5;
    typedef typename cplx<TC>::t C;
    constexpr int N = S3::N, AT = S3::AT, AE = S3::AE;
    __shared__ double red[80];
    const int ch = blockIdx.x % S3::ACH, comp = blockIdx.x / S3::ACH, n = blockIdx.y + gridDim.y * blockIdx.z;
    if (n >= a.S) return;
    const size_t fb = ((size_t)comp * a.S + n) * N;
    const int i0 = ch * (AT * AE) + threadIdx.x;
    const bool haveH = CORR || PASS == 3 || (PASS == 0 && !a.fk_given);
    TY *Y = (TY *)a.y;
    constexpr int NR = PASS == 0 ? NH - 1 : CORR ? 1 : 0;
    TY yv[AE];
    C hv[AE];
    TH fr[AE][NR > 0 ? NR : 1], fkg[AE];
#pragma unroll
    for (int k = 0; k < AE; k++) {
        const int i = i0 + k * AT;
        if (i < N) {
            yv[k] = Y[fb + i];
            if (haveH) hv[k] = H[fb + i];
            if (PASS == 0) {
#pragma unroll
                for (int j = 0; j < NR; j++) fr[k][j] = ld_stream((const TH *)a.slot[j] + fb + i);
                if (!haveH) fkg[k] = ld_stream((const TH *)a.slot[NH - 1] + fb + i);
            } else if (CORR) {
                fr[k][0] = ld_stream((const TH *)a.slot[NH - 2] + fb + i);
            }
        }
    }
    const double s = sc[n], E = haveH ? a.qpe[n] : 0.0, dt = a.dt, sn = PASS == 5 ? scn[n] : 1.0;
    double nrm = 0.0;
#pragma unroll
    for (int k = 0; k < AE; k++) {
        const int i = i0 + k * AT;
        if (i >= N) continue;
        double2 y0 = to_d(yv[k]);
        y0.x *= s; y0.y *= s;
        double2 fk = make_double2(0.0, 0.0), out = y0;
        if (haveH) {
            const double2 h = to_d(hv[k]);
            fk.x = h.x * s - E * y0.x;
            fk.y = h.y * s - E * y0.y;
        } else if (PASS == 0) {
            fk = to_d(fkg[k]);
        }
        if (PASS == 3) {
            ((TH *)a.slot[NH - 1])[fb + i] = from_d<TH>(fk);
            continue;
        }
        if (PASS == 0) {
            typedef Abm<NH> A;
            double2 sb = make_double2(fk.x * A::b(0), fk.y * A::b(0)), sa = make_double2(fk.x * A::a(0), fk.y * A::a(0));
#pragma unroll
            for (int j = 1; j < NH; j++) {
                const double2 fj = to_d(fr[k][j - 1]);
                sb.x += fj.x * A::b(j); sb.y += fj.y * A::b(j);
                if (j < A::na) { sa.x += fj.x * A::a(j); sa.y += fj.y * A::a(j); }
            }
            out.x = y0.x + dt * sb.y; out.y = y0.y - dt * sb.x;
            const double2 P = make_double2(y0.x + dt * sa.y, y0.y - dt * sa.x);
            if (haveH) st_stream((TH *)a.slot[NH - 1] + fb + i, from_d<TH>(fk));
            st_stream((TH *)a.slot[NH - 2] + fb + i, from_d<TH>(P));
        } else if (CORR) {
            const double2 P = to_d(fr[k][0]);
            out.x = dt * fk.y * Abm<NH>::c + P.x;
            out.y = -dt * fk.x * Abm<NH>::c + P.y;
        }
        if (PASS == 5) {
            Y[fb + i] = from_d<TY>(make_double2(out.x * sn, out.y * sn));
            continue;
        }
        nrm += out.x * out.x + out.y * out.y;
        if (PASS != 2 && PASS != 4) Y[fb + i] = from_d<TY>(out);
    }
    if (PASS != 3 && PASS != 5) {
        nrm = block_sum(nrm, red);
        if (threadIdx.x == 0) npart[(size_t)n * (2 * S3::ACH) + comp * S3::ACH + ch] = nrm;
    }
}

/* y <- scale y, scale <- 1 (the caller's states are normalised) */
template <typename TY>
__global__ void __launch_bounds__(S3::AT) k3s_rescale(TY *Y, const double *__restrict__ sc, int S)
{
    constexpr int N = S3::N;
    const int ch = blockIdx.x % S3::ACH, comp = blockIdx.x / S3::ACH, n = blockIdx.y + gridDim.y * blockIdx.z;
    if (n >= S) return;
    const size_t fb = ((size_t)comp * S + n) * N;
    const double s = sc[n];
#pragma unroll
    for (int k = 0; k < S3::AE; k++) {
        const int i = ch * (S3::AT * S3::AE) + k * S3::AT + threadIdx.x;
        if (i < N) {
            const double2 y = to_d(Y[fb + i]);
            Y[fb + i] = from_d<TY>(make_double2(y.x * s, y.y * s));
        }
    }
}
__global__ void k3s_fill(double *p, double v, int n)
{
    const int i = threadIdx.x + blockIdx.x * blockDim.x;
    if (i < n) p[i] = v;
}

/* nu, rho_a, rho_b at 128 points, summed over one chunk of states in registers; slots
 * [chunk][nu (2N), rho_a, rho_b] */
template <typename TY>
__global__ void __launch_bounds__(128) k3s_dens_points(int S, int nchunk, const TY *__restrict__ Y, const double *__restrict__ sc,
                                                       const double *__restrict__ occ, const double *__restrict__ wcnt,
                                                       double *slots)
{
    constexpr int N = S3::N;
    const int p = blockIdx.x * 128 + threadIdx.x;
    if (p >= N) return;
    const int s0 = (int)((long long)S * blockIdx.y / nchunk), s1 = (int)((long long)S * (blockIdx.y + 1) / nchunk);
    const size_t SN = (size_t)S * N;
    double nre = 0.0, nim = 0.0, ra = 0.0, rb = 0.0;
#pragma unroll 4
    for (int s = s0; s < s1; s++) {
        const double f = occ[s], c2 = sc[s] * sc[s] * wcnt[s];
        const double fa = f * c2, fb = (1.0 - f) * c2, fn = (1.0 - 2.0 * f) * 0.5 * c2;
        const double2 u = to_d(Y[(size_t)s * N + p]), v = to_d(Y[SN + (size_t)s * N + p]);
        nre += (u.x * v.x + u.y * v.y) * fn;
        nim += (u.y * v.x - u.x * v.y) * fn;
        ra += (u.x * u.x + u.y * u.y) * fa;
        rb += (v.x * v.x + v.y * v.y) * fb;
    }
    double *ds = slots + (size_t)blockIdx.y * 4 * N;
    ds[2 * p] = nre;
    ds[2 * p + 1] = nim;
    ds[2 * (size_t)N + p] = ra;
    ds[3 * (size_t)N + p] = rb;
}

/* totals of one point of a line over the re and im threads (adjacent lanes): tau is summed by
 * the im thread and j by the re thread, so each adds one word of its accumulator */
template <typename TC>
__device__ __forceinline__ double pair_tau(TC f, TC l, unsigned lanes = 0xffffffffu)
{
    const double t = (double)f * (double)l;
    return t + __shfl_xor_sync(lanes, t, 1);
}
template <typename TC>
__device__ __forceinline__ double pair_j(TC f, TC d, int c, unsigned lanes = 0xffffffffu)
{
    /* Im(psi* d psi) = re d im - im d re */
    const TC o = __shfl_xor_sync(lanes, f, 1);
    const double t = (c ? 1.0 : -1.0) * (double)o * (double)d;
    return t + __shfl_xor_sync(lanes, t, 1);
}

/* tau_tmp and j along the y and z lines of one (component, x-plane) over one chunk of states;
 * slots [chunk][component][tau, j_y, j_z][N].  Accumulators in shared memory: A[row][2 z + {j_y,
 * tau}] and B[row][z] = j_z, rows padded to odd lengths. */
template <typename TC> struct S3DensSmem {
    typedef typename cplx<TC>::t C;
    static constexpr size_t plane = (size_t)S3::PL * sizeof(C);
    static constexpr size_t pbytes = plane + 3 * (size_t)S3::PL * sizeof(double);
    static constexpr size_t xbytes = (size_t)4 * NX * S3::QB * sizeof(double);
};
template <typename TY, typename TC>
__global__ void __launch_bounds__(S3::LT) k3s_dens_plane(int S, int nchunk, const TY *__restrict__ Y, const double *__restrict__ sc,
                                                         const double *__restrict__ occ, const double *__restrict__ wcnt,
                                                         double *slots)
{
    typedef typename cplx<TC>::t C;
    constexpr int N = S3::N, NYZ = S3::NYZ, LT = S3::LT, PITCH = S3::PITCH, PL = S3::PL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *P = (C *)smem_raw;
    TC *Pr = (TC *)P;
    double *A = (double *)(smem_raw + S3DensSmem<TC>::plane), *B = A + 2 * PL;
    const int t = threadIdx.x, line = t >> 1, c = t & 1;
    const int pr = (int)(blockIdx.x % (2 * NX)), chunk = (int)(blockIdx.x / (2 * NX));
    const int comp = pr / NX, x = pr - comp * NX;
    for (int i = t; i < 3 * PL; i += LT) A[i] = 0.0;
    const int s0 = (int)((long long)S * chunk / nchunk), s1 = (int)((long long)S * (chunk + 1) / nchunk);
    const double jsgn = comp ? -1.0 : 1.0;
    for (int n = s0; n < s1; n++) {
        const size_t base = ((size_t)comp * S + n) * N + (size_t)x * NYZ;
        const double f0 = occ[n], w = (comp ? 1.0 - f0 : f0) * wcnt[n] * (sc[n] * sc[n]), wj = w * jsgn;
        if (t == 0 && n + 1 < s1) prefetch_l2(Y + base + N, NYZ * sizeof(TY));
        __syncthreads();
#pragma unroll 8
        for (int i = t; i < NYZ; i += LT) {
            const TY a = Y[base + i];
            C z; z.x = a.x; z.y = a.y;
            P[(i / NZ) * PITCH + i % NZ] = z;
        }
        __syncthreads();
        {
            /* every lane runs the line (the exchanges take whole warps); only real lines add */
            const bool on = line < NY;
            const int r = on ? line : 0;
            TC f[NZ], l[NZ];
#pragma unroll
            for (int j = 0; j < NZ; j++) f[j] = Pr[2 * (r * PITCH + j) + c];
            circ::line_op<circ::LAP, 2, NZ>(f, l);
#pragma unroll
            for (int j = 0; j < NZ; j++) {
                const double v = pair_tau(f[j], l[j]);
                if (on && c) A[2 * (r * PITCH + j) + 1] += v * w;
            }
            circ::line_op<circ::DER, 2, NZ>(f, l);
#pragma unroll
            for (int j = 0; j < NZ; j++) {
                const double v = pair_j(f[j], l[j], c);
                if (on && !c) B[r * PITCH + j] += v * wj;
            }
        }
        __syncthreads();
        {
            const bool on = line < NZ;
            const int r = on ? line : 0;
            TC f[NY], l[NY];
#pragma unroll
            for (int j = 0; j < NY; j++) f[j] = Pr[2 * (j * PITCH + r) + c];
            circ::line_op<circ::LAP, 1, NY>(f, l);
#pragma unroll
            for (int j = 0; j < NY; j++) {
                const double v = pair_tau(f[j], l[j]);
                if (on && c) A[2 * (j * PITCH + r) + 1] += v * w;
            }
            circ::line_op<circ::DER, 1, NY>(f, l);
#pragma unroll
            for (int j = 0; j < NY; j++) {
                const double v = pair_j(f[j], l[j], c);
                if (on && !c) A[2 * (j * PITCH + r)] += v * wj;
            }
        }
    }
    __syncthreads();
    double *ds = slots + ((size_t)chunk * 2 + comp) * 3 * N + (size_t)x * NYZ;
    for (int i = t; i < NYZ; i += LT) {
        const int o = (i / NZ) * PITCH + i % NZ;
        ds[i] = A[2 * o + 1];
        ds[(size_t)N + i] = A[2 * o];
        ds[2 * (size_t)N + i] = B[o];
    }
}

/* tau_tmp and j_x along the x lines of a block of columns of both components over one chunk of
 * states; slots [chunk][component][tau, j_x][N] */
template <typename TY, typename TC>
__global__ void __launch_bounds__(2 * S3::XL) k3s_dens_x(int S, int nchunk, const TY *__restrict__ Y, const double *__restrict__ sc,
                                                         const double *__restrict__ occ, const double *__restrict__ wcnt,
                                                         double *slots)
{
    constexpr int N = S3::N, NYZ = S3::NYZ, QB = S3::QB, XL = S3::XL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int qb = (int)(blockIdx.x % S3::NQB), chunk = (int)(blockIdx.x / S3::NQB), q0 = qb * QB;
    const int comp = threadIdx.x / XL, lane = threadIdx.x - comp * XL, q = lane >> 1, c = lane & 1;
    double *A = (double *)smem_raw + (size_t)comp * 2 * NX * QB;   /* [x][2 q + {j, tau}], own word */
    for (int x = 0; x < NX; x++) A[2 * (x * QB + q) + c] = 0.0;
    const int s0 = (int)((long long)S * chunk / nchunk), s1 = (int)((long long)S * (chunk + 1) / nchunk);
    const double jsgn = comp ? -1.0 : 1.0;
    for (int n = s0; n < s1; n++) {
        const TC *yr = (const TC *)Y + 2 * (((size_t)comp * S + n) * N + q0 + q) + c;
        const double f0 = occ[n], w = (comp ? 1.0 - f0 : f0) * wcnt[n] * (sc[n] * sc[n]), wj = w * jsgn;
        if (n + 1 < s1)
            for (int r = lane; r < NX; r += XL) prefetch_l2(Y + ((size_t)comp * S + n + 1) * N + (size_t)r * NYZ + q0, QB * sizeof(TY));
        TC f[NX], l[NX];
#pragma unroll
        for (int x = 0; x < NX; x++) f[x] = yr[(size_t)2 * x * NYZ];
        circ::line_op<circ::LAP, 0, NX>(f, l);
#pragma unroll
        for (int x = 0; x < NX; x++) {
            const double v = pair_tau(f[x], l[x], S3::XM);
            if (c) A[2 * (x * QB + q) + 1] += v * w;
        }
        circ::line_op<circ::DER, 0, NX>(f, l);
#pragma unroll
        for (int x = 0; x < NX; x++) {
            const double v = pair_j(f[x], l[x], c, S3::XM);
            if (!c) A[2 * (x * QB + q)] += v * wj;
        }
    }
    double *ds = slots + ((size_t)chunk * 2 + comp) * 2 * N + q0 + q + (c ? 0 : (size_t)N);
    for (int x = 0; x < NX; x++) ds[(size_t)x * NYZ] = A[2 * (x * QB + q) + c];
}

/* densities from the slots of the three kernels, in fixed order (pca_dens.cu:13-198); without
 * gradients only nu and rho, the rest 0 */
__global__ void __launch_bounds__(256) k3s_dens_reduce(const double *sp, int gp, const double *sy, int gy, const double *sx, int gx,
                                                       double *dens, int full, double inv_lperp)
{
    constexpr int N = S3::N;
    const int i = threadIdx.x + blockIdx.x * blockDim.x;
    if (i >= 12 * N) return;
    auto total = [&](int w) -> double {
        double s = 0.0;
        if (w < 2 * N) {
            for (int k = 0; k < gp; k++) s += sp[(size_t)k * 4 * N + w];
            return s;
        }
        const int b = (w - 2 * N) / N, p = w - (2 + b) * N, comp = b >= 5 ? 1 : 0, r = b - 5 * comp;   /* rho tau jx jy jz */
        if (r == 0) {
            for (int k = 0; k < gp; k++) s += sp[(size_t)k * 4 * N + (size_t)(2 + comp) * N + p];
            return s;
        }
        if (!full) return 0.0;
        if (r == 1 || r == 2)
            for (int k = 0; k < gx; k++) s += sx[((size_t)(2 * k + comp) * 2 + (r - 1)) * N + p];
        if (r != 2)
            for (int k = 0; k < gy; k++) s += sy[((size_t)(2 * k + comp) * 3 + (r == 1 ? 0 : r - 2)) * N + p];
        return s;
    };
    double s = total(i);
#ifdef SPINSYMMETRY_MODE
    /* both spin channels take the sum of the u and v contributions, nu counts twice */
    if (i < 2 * N) s *= 2.0;
    else s += total(i < 7 * N ? i + 5 * N : i - 5 * N);
#endif
    dens[i] = s * inv_lperp;
}

/* ---------------------------------------------------------------------------------------
 * derivatives of the O(N) real fields, one thread per line, one launch per axis for all fields
 * (the transforms of wtd_fft3d.cuh took 40 launches for the coefficients and 10 for tau, which is
 * most of a half step of few states)
 * -------------------------------------------------------------------------------------*/
template <int AX> struct S3Line {
    static constexpr int n = AX == 0 ? NX : AX == 1 ? NY : NZ, lines = S3::N / n;
    int base;
    static constexpr int st = AX == 0 ? S3::NYZ : AX == 1 ? NZ : 1;
    __device__ __forceinline__ S3Line(int l) { base = AX == 0 ? l : AX == 1 ? (l / NZ) * S3::NYZ + l % NZ : l * NZ; }
};
/* lap(alpha_s)/4 (blockIdx.y = 0, 1) and -div(A_s)/2 (2, 3): axis AX's part, added to the earlier */
template <int AX>
__global__ void __launch_bounds__(64) k3s_coef_axis(double *cf)
{
    typedef S3Line<AX> L;
    const int l = threadIdx.x + blockIdx.x * 64, o = blockIdx.y, s = o & 1;
    if (l >= L::lines) return;
    const L line(l);
    const double *src = cf + (size_t)(o < 2 ? CF_ALA + s : (s ? CF_ABX : CF_AAX) + AX) * S3::N + line.base;
    double *dst = cf + (size_t)(o < 2 ? CF_NA + s : CF_CJA + s) * S3::N + line.base;
    double v[L::n];
    circ::MemLine<double> f{src, L::st};
    if (o < 2) circ::line_from<circ::LAP, AX, L::n>(f, v);
    else circ::line_from<circ::DER, AX, L::n>(f, v);
    const double w = o < 2 ? 0.25 : -0.5;
#pragma unroll
    for (int j = 0; j < L::n; j++) dst[j * L::st] = AX > 0 ? dst[j * L::st] + w * v[j] : w * v[j];
}
/* tau_s = max(0, lap(rho_s)/2 - tau_s) (pca_dens.cu:275-338), the laplacian gathered in tmp over the
 * axes; blockIdx.y = spin */
template <int AX>
__global__ void __launch_bounds__(64) k3s_tau_axis(double *dens, double *tmp)
{
    typedef S3Line<AX> L;
    const int l = threadIdx.x + blockIdx.x * 64, s = blockIdx.y;
    if (l >= L::lines) return;
    const L line(l);
    double v[L::n], *t = tmp + (size_t)s * S3::N + line.base;
    circ::MemLine<double> f{dens + (size_t)(s ? 7 : 2) * S3::N + line.base, L::st};
    circ::line_from<circ::LAP, AX, L::n>(f, v);
    if (AX < 2) {
#pragma unroll
        for (int j = 0; j < L::n; j++) t[j * L::st] = AX > 0 ? t[j * L::st] + v[j] : v[j];
    } else {
        double *tau = dens + (size_t)(s ? 8 : 3) * S3::N + line.base;
#pragma unroll
        for (int j = 0; j < L::n; j++) {
            const double r = 0.5 * (t[j * L::st] + v[j]) - tau[j * L::st];
            tau[j * L::st] = r < 0.0 ? 0.0 : r;
        }
    }
}

#endif /* CODEDIM == 3 */
#endif
