/*
 * vh_physics.cuh -- per-cell device physics of the KT RK2 step, in FP64 and in
 * the reference's floating-point operation order (the library is compiled
 * with --fmad=false, so nothing below is fused unless written as fma()).
 *
 * Each function names the reference code it reproduces (file:line in
 * derekeverett/cpu-vh).  The state lives in padded SoA arrays (stride L
 * doubles between components) indexed i + ncx*(j + ncy*k).
 */
#ifndef VH_PHYSICS_CUH
#define VH_PHYSICS_CUH

#include "vh_math.cuh"

namespace vh {

/* error codes raised on the device (match VH_ERR_* in vh_b200.h) */
constexpr int kErrNan = 4;

struct DevEos {
    int kind;                 /* 0 conformal, 1 table */
    double a;                 /* conformal e = a T^4 */
    const double *p_tb;       /* tabulated P(e) [fm^-4] */
    const double *T_tb;       /* tabulated T(e) [fm^-1] */
    int e_length;
    double e_min, e_spacing;
    double inv_spacing;       /* RN(1/e_spacing), for div_rcp */
    double cs2_third_hi;      /* eos_cs2 is exactly 1/3 for e <= this (HostEos::cs2_third_bound) */
    unsigned direct;          /* flow_pair's root solve: 2^-60 <= |e| with a high word less than `direct` above that
                                 of 2^-60 is below min(2^60, cs2_third_hi); 0: not for this table */
    int ranged;               /* the table's e_min and e_spacing lie where eos_interp_direct is exact */
    PowfTab pq;               /* host-exact powf(x, 0.25) */
    const int *stop;          /* the event's device error code (or null): see e_bisect_table */
};

struct DevErr {
    int *code;                /* first error code, 0 if none */
    long long *cell;          /* padded index of the first failing cell */
    int *step;                /* step counter at the time */
};

__device__ __forceinline__ void raise_error(const DevErr &E, int code, long long cell, int step)
{
    if (atomicCAS(E.code, 0, code) == 0) { *E.cell = cell; *E.step = step; }
}

/* ---------------------------------------------- division, shared divisor */
/* IEEE a/b, kept out of line: the fallback of div_rcp */
static __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }

/* The correctly rounded quotient a/b given y = RN(1/b), by Markstein's
 * theorem (P. Markstein, IBM J. Res. Dev. 34(1), 1990; Muller et al.,
 * Handbook of Floating-Point Arithmetic, ch. 4): q0 = RN(a*y) is within one
 * ulp of a/b, r = a - q0*b is exact with an FMA, and RN(q0 + r*y) = RN(a/b).
 * One reciprocal then serves every division by the same b at the cost of a
 * multiply and two FMAs each -- bit-identical to `a / b`.  The range test
 * (|a|, |y| >= 2^-960 and 2^-960 <= |q0| < 2^1000) reads the high words
 * with integer operations.  A zero numerator over a finite b gives q0 = a * y =
 * +-0 with the sign of a XOR the sign of b, which is a / b exactly (zero
 * numerators are common: velocity and viscous components that are still
 * exactly 0).  Non-finite, huge or near-subnormal operands, where the
 * exactness argument needs more care, take the IEEE division. */
__device__ __forceinline__ double div_rcp(double a, double b, double y)
{
    constexpr unsigned kLo = 0x03f00000u;      /* high word of 2^-960 */
    constexpr unsigned kHi = 0x7e700000u;      /* high word of 2^1000 */
    const double q0 = a * y;
    const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu;
    const unsigned hq = (unsigned)__double2hiint(q0) & 0x7fffffffu;
    const unsigned hy = (unsigned)__double2hiint(y) & 0x7fffffffu;
    if (ha >= kLo && hq >= kLo && hq < kHi && hy >= kLo) {
        const double r = fma(-q0, b, a);
        return fma(r, y, q0);
    }
    if ((ha | (unsigned)__double2loint(a)) == 0u && hq < 0x7ff00000u) return q0;
    return div_ieee(a, b);
}

/* ------------------------------------------------------------------ EoS */
/* EquationOfState.cpp:329-360 */
__device__ __forceinline__ double eos_interp(const DevEos &E, double ed, const double *tb)
{
    int idx = (int)div_rcp(ed - E.e_min, E.e_spacing, E.inv_spacing);
    idx = (E.e_length - 2 < idx) ? E.e_length - 2 : idx;   /* std::min(N_e - 2, idx) */
    idx = (idx < 0) ? 0 : idx;                              /* std::max(0, idx)       */
    const double frac = div_rcp(ed - (idx * E.e_spacing + E.e_min), E.e_spacing, E.inv_spacing);
    return __ldg(tb + idx) * (1. - frac) + __ldg(tb + idx + 1) * frac;
}
/* std::max(1.e-15, f): (1e-15 < f) ? f : 1e-15 */
__device__ __forceinline__ double floor15(double f) { return (1.e-15 < f) ? f : 1.e-15; }

template <int EOS>
__device__ __forceinline__ double eos_p(const DevEos &E, double ed)          /* EquationOfState.cpp:44-107 */
{
    if (EOS == 1) return floor15(eos_interp(E, ed, E.p_tb));
    return ed / 3.;
}
template <int EOS>
__device__ __forceinline__ double eos_cs2(const DevEos &E, double ed)        /* EquationOfState.cpp:109-160 */
{
    if (EOS == 1) {
        const double v_min = 0.01, v_max = 1. / 3.;
        if (ed <= E.cs2_third_hi) return v_max;    /* the clamp's value, proven for this table */
        double pp = eos_p<1>(E, ed);
        double p_r = eos_p<1>(E, ed + E.e_spacing);
        double v = E.e_spacing / (p_r - pp);
        v = (v < v_max) ? v : v_max;            /* std::min(v_max, v) */
        return (v_min < v) ? v : v_min;         /* std::max(v_min, v) */
    }
    return 1. / 3.;
}
template <int EOS>
__device__ __forceinline__ double eos_T(const DevEos &E, double ed)          /* EquationOfState.cpp:162-199 */
{
    if (EOS == 1) return floor15(eos_interp(E, ed, E.T_tb));
    return (double)powf_quarter(__double2float_rn(ed / E.a), E.pq);
}

/* --------------------------------------------------------- limiter */
/* FluxLimiter.cpp:14-32, generalised minmod with sign(0) = +1:
 * (sign(x) + sign(y)) * min(|x|, |y|) / 2, evaluated without the integer
 * sum and its conversion.  The factor is +-2 or 0, and 2m / 2 = m exactly
 * for m = min(|x|, |y|) below 2^1023 (no overflow in 2m), so the result is
 * +-m when the signs agree and 0 * m (+0, or NaN for m = inf) when they
 * differ -- the same value, sign of zero and NaN cases included. */
__device__ __forceinline__ double minmod(double x, double y)
{
    const bool nx = x < 0, ny = y < 0;
    const double m = fmin(fabs(x), fabs(y));
    return (nx == ny) ? (nx ? -m : m) : 0.0 * m;
}
__device__ __forceinline__ double approx_deriv(double th, double x, double y, double z)
{
    double l = th * (y - x);
    double c = (z - x) / 2.0;
    double r = th * (z - y);
    return minmod(l, minmod(c, r));
}

/* approx_deriv with the three differences' common sign taken from their sign
 * bits and the minimum of their magnitudes from their bit patterns (which
 * order as the magnitudes do): all negative -> -m, none negative -> m, else
 * +0.  A difference of -0 counts as negative here and not there, but then m = 0
 * and both give +0 (the FMA adds +0).  theta is finite (limiter_ranged), so a
 * difference is a NaN only where a value is none or infinite; its sign, which
 * counts here and not there, may then give another slope, but the state is no
 * state and its step raises the error either way.  one: the high word of the factor
 * on m, 0x3ff00000 for 1, 0x3fe00000 for 1/2 (RN(m/2) as approx_deriv / 2). */
__device__ __forceinline__ double limited(double th, double x, double y, double z, int one)
{
    const double l = th * (y - x), c = (z - x) / 2.0, r = th * (z - y);
    const long long il = __double_as_longlong(l), ic = __double_as_longlong(c), ir = __double_as_longlong(r);
    const long long msk = 0x7fffffffffffffffLL;
    const long long m = min(il & msk, min(ic & msk, ir & msk));
    const int hl = (int)(il >> 32), hc = (int)(ic >> 32), hr = (int)(ir >> 32);
    const int hi = ((hl & hc & hr) < 0) ? (one | (int)0x80000000) : ((hl | hc | hr) >= 0) ? one : 0;
    return fma(__longlong_as_double(m), __hiloint2double(hi, 0), 0.0);
}

/* -------------------------------------------------------- inversion */
/* EnergyMomentumTensor.cpp:48-111: the bisection the tabulated-EoS root solve
 * falls back to when Newton has not converged in 10^4 iterations.  Out of
 * line: no valid state here reaches it, and every caller shares one copy.
 * Once the event's device has flagged an error, the bisection gives up after
 * 64 iterations: the state is then invalid (the reference exits at its first
 * NaN), and the cells of a garbage state would each spend its 10^6
 * iterations before the host reads the error.  The flag is read through L2
 * (another block may have just set it). */
static __device__ __noinline__ double e_bisect_table(const DevEos &E, double ePrev, double M0, double M, double Pi)
{
    double e_lo = 0.0, e_mid = ePrev, e_hi = 2.0 * (ePrev + 1.0);
    for (int j = 0; j < 1000000; ++j) {                            /* MAX_ITERS_BI */
        if ((j & 63) == 63 && E.stop && *(const volatile int *)E.stop != 0) return ePrev;
        double p_lo = eos_p<1>(E, e_lo), p_mid = eos_p<1>(E, e_mid), p_hi = eos_p<1>(E, e_hi);
        double c_lo = p_lo / e_lo, c_mid = p_mid / e_mid, c_hi = p_hi / e_hi;
        double A_lo = M0 * (1.0 - c_lo) + Pi, A_mid = M0 * (1.0 - c_mid) + Pi, A_hi = M0 * (1.0 - c_hi) + Pi;
        double B = M0 * (M0 + Pi) - M;
        double H_lo = (double)sqrtf(fabsf(__double2float_rn(A_lo * A_lo + 4 * c_lo * B)));
        double H_mid = (double)sqrtf(fabsf(__double2float_rn(A_mid * A_mid + 4 * c_mid * B)));
        double H_hi = (double)sqrtf(fabsf(__double2float_rn(A_hi * A_hi + 4 * c_hi * B)));
        double f_lo = e_lo + (A_lo - H_lo) / (2 * c_lo);
        double f_mid = e_mid + (A_mid - H_mid) / (2 * c_mid);
        double f_hi = e_hi + (A_hi - H_hi) / (2 * c_hi);
        if ((e_hi - e_lo) < (1.0e-3 * e_hi) / 2.0) return e_mid;
        if (f_lo * f_mid < 0.0) { e_hi = e_mid; e_mid = (e_lo + e_hi) / 2.0; }
        else if (f_mid * f_hi < 0.0) { e_lo = e_mid; e_mid = (e_lo + e_hi) / 2.0; }
    }
    return ePrev;
}

/* One Newton iteration of EnergyMomentumTensor.cpp:22-44 from e0: the next
 * iterate, whether f/f' is NaN, and whether the float-truncated convergence
 * test (:41) passes. */
__device__ __forceinline__ double e_newton_iter(const DevEos &E, double e0, double M0, double M, double Pi,
                                                bool &nan_step, bool &conv)
{
    double pp = eos_p<1>(E, e0);
    double cs2 = eos_cs2<1>(E, e0);
    double cst2 = pp / e0;
    double A = M0 * (1.0 - cst2) + Pi;
    double B = M0 * (M0 + Pi) - M;
    double H = (double)sqrtf(fabsf(__double2float_rn(A * A + 4 * cst2 * B)));
    double D = (A - H) / (2 * cst2);
    double f = e0 + D;
    double fp = 1.0 - ((cs2 - cst2) * (B + D * H - ((cs2 - cst2) * cst2 * D * M0) / e0)) / (cst2 * e0 * H);
    double q = f / fp;
    double e = e0 - q;
    nan_step = isnan(q);
    conv = (double)fabsf(__double2float_rn(e - e0)) <= 1.0e-3 * (double)fabsf(__double2float_rn(e));
    return e;
}

/* EnergyMomentumTensor.cpp:22-111, the tabulated-EoS root solve: Newton from
 * ePrev, bisection if Newton does not converge. */
__device__ __forceinline__ double e_newton_table_body(const DevEos &E, double ePrev, double M0, double M, double Pi, bool &bad)
{
    double e0 = ePrev;
    for (int j = 0; j < 10000; ++j) {                              /* MAX_ITERS_NR */
        bool nan_step, conv;
        double e = e_newton_iter(E, e0, M0, M, Pi, nan_step, conv);
        if (nan_step) { bad = true; return ePrev; }
        if (conv) return e;
        e0 = e;
    }
    return e_bisect_table(E, ePrev, M0, M, Pi);
}

/* the same from iterate e0 of iteration j0 on, out of line: a solve that is
 * still going after the few iterations it usually takes.  It gives up (false)
 * where energy_direct's own loop does: a solve that ends in the bisection, which
 * may run for a second, is then the plain form's alone and not run twice */
constexpr int kDirectIters = 100;
static __device__ __noinline__ bool e_newton_rest(const DevEos &E, double e0, int j0, double M0, double M, double Pi, double &e)
{
    for (int j = j0; j < kDirectIters; ++j) {
        bool nan_step, conv;
        e = e_newton_iter(E, e0, M0, M, Pi, nan_step, conv);
        if (nan_step) return false;
        if (conv) return true;
        e0 = e;
    }
    return false;
}

/* The root solve as a call (one copy of the loop for a long kernel whose
 * instruction footprint matters) or inlined (short phase kernels). */
static __device__ __noinline__ double e_newton_table(const DevEos &E, double ePrev, double M0, double M, double Pi, bool &bad)
{
    return e_newton_table_body(E, ePrev, M0, M, Pi, bad);
}

/* EnergyMomentumTensor.cpp:22-115: energy density from M0, M, Pi; the
 * conformal closed form (:113) truncates through float. */
template <int EOS, bool INL = false>
__device__ __forceinline__ double e_from_conserved(const DevEos &E, double ePrev, double M0, double M, double Pi, bool &bad)
{
    if (EOS == 0) {
        float h = sqrtf(fabsf(__double2float_rn(4 * M0 * M0 - 3 * M)));
        return (double)fabsf(__double2float_rn((double)h - M0));
    }
    if (INL) return e_newton_table_body(E, ePrev, M0, M, Pi, bad);
    return e_newton_table(E, ePrev, M0, M, Pi, bad);
}

struct Prim { double e, p, ut, ux, uy, un; };

/* EnergyMomentumTensor.cpp:117-233, from the five combinations it uses
 * (M0 = ttt - pitt, M1..M3 = tt^i - pit^i, Pi). */
template <int EOS, bool INL = false>
__device__ __forceinline__ Prim infer(const DevEos &E, double t, double M0, double M1, double M2, double M3,
                                      double Pi, double ePrev, bool &bad)
{
    Prim r;
    double M = M1 * M1 + M2 * M2 + t * t * M3 * M3;
    if (ePrev <= 0.1) r.e = M0 - M / M0;
    else r.e = e_from_conserved<EOS, INL>(E, ePrev, M0, M, Pi, bad);
    if (isnan(r.e)) bad = true;
    r.p = eos_p<EOS>(E, r.e);
    if (r.e < 1.e-7) { r.e = 1.e-7; r.p = 1.e-7; }
    double P = r.p + Pi;
    double Einv = 1.0 / (r.e + P);
    r.ut = (double)sqrtf(fabsf(__double2float_rn((M0 + P) * Einv)));
    double E2 = Einv / r.ut;
    r.ux = M1 * E2;
    r.uy = M2 * E2;
    r.un = M3 * E2;
    if (r.ut > 1.0e3) { r.ut = 1.0; r.ux = 0.0; r.uy = 0.0; r.un = 0.0; }
    return r;
}

/* ------------------------------------------------------------------
 * The same inversion for the two half-site states of a face, side by side and
 * without the divisions' branches (rcp_rn, div_rn, sqrt_rn): what a flux needs
 * of each state is u^tau, one velocity component and RN(1/u^tau).  Two
 * independent Newton chains per thread overlap where one leaves the FP64 pipe
 * idle between dependent operations.  Every value is e_newton_iter's and
 * infer's, in their operation order, and every quotient is the correctly
 * rounded one, so the result has infer's bits.  M1..M3 and Pi are formed from
 * values that pass state_ranged; where another operand leaves the range the
 * exactness needs, flow_pair returns false and the caller runs infer.
 * ------------------------------------------------------------------ */
struct Flow { double ut, v, y; };       /* u^tau, u^dir, RN(1/u^tau) */

template <bool MIXED = false>
__device__ __forceinline__ double eos_interp_direct(const DevEos &E, double ed, const double *tb)
{
    /* ed - e_min and ed minus a node are 0 or far above 2^-900 for ed >=
     * 2^-100 and a table whose e_min is 0 or at least 2^-100 */
    int idx = (int)div_rn(ed - E.e_min, E.e_spacing, E.inv_spacing);
    idx = (E.e_length - 2 < idx) ? E.e_length - 2 : idx;
    idx = (idx < 0) ? 0 : idx;
    const double frac = div_rn(ed - (idx * E.e_spacing + E.e_min), E.e_spacing, E.inv_spacing);
    const double lo = __ldg(tb + idx), hi = __ldg(tb + idx + 1);
    /* the mixed translation unit contracts eos_interp's sum this way */
    if (MIXED) return fma(lo, 1. - frac, hi * frac);
    return lo * (1. - frac) + hi * frac;
}

/* the FP32 square root as infer takes it: correctly rounded, or in the mixed
 * translation unit the fast one its sqrtf compiles to (branch-free anyway) */
template <bool MIXED>
__device__ __forceinline__ float root32(float x)
{
    if constexpr (MIXED) return sqrtf(x);
    else return sqrt_rn(x);
}

/* the energy density of N states (e_from_conserved, or infer's closed form
 * below ePrev = 0.1); M = M1^2 + M2^2 + t^2 M3^2.  REST: a solve still going
 * after 8 iterations (one state in a steep gradient of a coarse lattice) ends
 * out of line, alone; the call costs the line-piece kernels registers (mixed
 * 131x131x61 4 %), so only the fused stage, whose time is its slowest thread,
 * takes it (21x21x9: 100 -> 84 us per step, mixed 91 -> 77) */
template <int EOS, int N, bool MIXED, bool REST = false>
__device__ __forceinline__ bool energy_direct(const DevEos &E, const double (&M0)[N], const double (&M)[N],
                                              const double (&Pi)[N], double ePrev, double (&ef)[N])
{
    bool ok = true;
#pragma unroll
    for (int s = 0; s < N; ++s) ok = ok && within<-60, 60>(M0[s]);
    if (ePrev <= 0.1) {
#pragma unroll
        for (int s = 0; s < N; ++s) {
            ok = ok && rcp_ok(M0[s]);
            ef[s] = M0[s] - div_rn(M[s], M0[s], rcp_rn(M0[s]));
        }
    } else if (EOS == 0) {
#pragma unroll
        for (int s = 0; s < N; ++s) {
            const float h2 = fabsf(__double2float_rn(4 * M0[s] * M0[s] - 3 * M[s]));
            ok = ok && in_range(h2);
            ef[s] = (double)fabsf(__double2float_rn((double)root32<MIXED>(h2) - M0[s]));
        }
    } else {
        double e0[N], B[N];
        bool done[N];
#pragma unroll
        for (int s = 0; s < N; ++s) {
            B[s] = M0[s] * (M0[s] + Pi[s]) - M[s];
            ef[s] = e0[s] = ePrev;
            done[s] = false;
        }
        const double cs2 = 1. / 3.;
        for (int j = 0; ok; ++j) {
            if (REST && j == 8) {
                /* few lanes are left, and of those mostly one state */
#pragma unroll
                for (int s = 0; s < N; ++s)
                    if (ok && !done[s]) ok = e_newton_rest(E, e0[s], j, M0[s], M[s], Pi[s], ef[s]);
                break;
            }
            if (j == kDirectIters) { ok = false; break; }
            bool all = true;
#pragma unroll
            for (int s = 0; s < N; ++s) {
                const double x = e0[s];
                /* (an iterate below zero, on its way down a steep gradient, is in
                 * range too: its p is the floor, 2^-49.8) */
                bool fine = ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((1023u - 60u) << 20) < E.direct && rcp_ok(x);
                const double pp = floor15(eos_interp_direct<MIXED>(E, x, E.p_tb));
                fine = fine && within<-50, 60>(pp);
                const double yx = rcp_rn(x);
                const double cst2 = div_rn(pp, x, yx);
                const double A = M0[s] * (1.0 - cst2) + Pi[s];
                const float h2 = fabsf(__double2float_rn(A * A + 4 * cst2 * B[s]));
                fine = fine && in_range(h2);
                const double H = (double)root32<MIXED>(h2);
                const double c2 = 2 * cst2;
                const double D = div_rn(A - H, c2, rcp_rn(c2));
                const double f = x + D;
                const double g = cs2 - cst2;
                const double w = g * cst2 * D * M0[s];
                const double num = g * (B[s] + D * H - div_rn(w, x, yx));
                const double den = cst2 * x * H;
                const double fp = 1.0 - div_rn(num, den, rcp_rn(den));
                const double q = div_rn(f, fp, rcp_rn(fp));
                fine = fine && rcp_ok(c2) && rcp_ok(den) && rcp_ok(fp) && in_range_abs(fp);
                const double e = x - q;
                const bool conv = (double)fabsf(__double2float_rn(e - x)) <= 1.0e-3 * (double)fabsf(__double2float_rn(e));
                if (!done[s]) {
                    ok = ok && fine;
                    ef[s] = e;
                    e0[s] = e;
                    done[s] = conv;
                }
                all = all && done[s];
            }
            if (all) break;
        }
    }
    return ok;
}

/* infer's e, p (floored), u^tau, RN(1/u^tau) and 1/((e + P) u^tau) from the
 * energy density; the last times M1..M3 is the velocity while u^tau <= 1e3 */
template <int EOS, bool MIXED>
__device__ __forceinline__ bool flow_direct(const DevEos &E, double M0, double Pi, double &e, double &p, double &ut,
                                            double &yu, double &E2)
{
    const bool low = e < 1.e-7;
    bool ok = low || in_range(e);
    p = (EOS == 1) ? floor15(eos_interp_direct<MIXED>(E, e, E.p_tb)) : div_rn(e, 3., 1. / 3.);
    if (low) { e = 1.e-7; p = 1.e-7; }
    const double P = p + Pi, W = e + P;
    const double Einv = rcp_rn(W);
    const float x = fabsf(__double2float_rn((M0 + P) * Einv));
    ok = ok && in_range_abs(W) && rcp_ok(W) && in_range(x);
    ut = (double)root32<MIXED>(x);          /* 24 significant bits: rcp_ok */
    yu = rcp_rn(ut);
    E2 = div_rn(Einv, ut, yu);
    return ok;
}

template <int EOS, bool MIXED = false, bool REST = false>
__device__ __forceinline__ bool flow_pair(const DevEos &E, double t, const double (&M0)[2], const double (&M1)[2],
                                          const double (&M2)[2], const double (&M3)[2], const double (&Pi)[2], int dir,
                                          double ePrev, Flow (&out)[2])
{
    double M[2], ef[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) M[s] = M1[s] * M1[s] + M2[s] * M2[s] + t * t * M3[s] * M3[s];
    bool ok = energy_direct<EOS, 2, MIXED, REST>(E, M0, M, Pi, ePrev, ef);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        double p, ut, yu, E2;
        ok = flow_direct<EOS, MIXED>(E, M0[s], Pi[s], ef[s], p, ut, yu, E2) && ok;
        double v = ((dir == 1) ? M1[s] : (dir == 2) ? M2[s] : M3[s]) * E2;
        if (ut > 1.0e3) { ut = 1.0; v = 0.0; yu = 1.0; }
        out[s].ut = ut;
        out[s].v = v;
        out[s].y = yu;
    }
    return ok;
}

/* infer for one state in the same form; false: run infer */
template <int EOS, bool MIXED = false>
__device__ __forceinline__ bool infer_direct(const DevEos &E, double t, double M0, double M1, double M2, double M3,
                                             double Pi, double ePrev, Prim &r)
{
    const double M0s[1] = {M0}, M[1] = {M1 * M1 + M2 * M2 + t * t * M3 * M3}, Pis[1] = {Pi};
    double ef[1], yu, E2;
    bool ok = energy_direct<EOS, 1, MIXED>(E, M0s, M, Pis, ePrev, ef);
    r.e = ef[0];
    ok = flow_direct<EOS, MIXED>(E, M0, Pi, r.e, r.p, r.ut, yu, E2) && ok;
    r.ux = M1 * E2;
    r.uy = M2 * E2;
    r.un = M3 * E2;
    if (r.ut > 1.0e3) { r.ut = 1.0; r.ux = 0.0; r.uy = 0.0; r.un = 0.0; }
    return ok;
}

/* flow_pair's two states through infer, one after the other */
template <int EOS>
__device__ __forceinline__ void flow_pair_plain(const DevEos &E, double t, const double (&M0)[2], const double (&M1)[2],
                                                const double (&M2)[2], const double (&M3)[2], const double (&Pi)[2],
                                                int dir, double ePrev, Flow (&out)[2], bool &bad)
{
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const Prim P = infer<EOS>(E, t, M0[s], M1[s], M2[s], M3[s], Pi[s], ePrev, bad);
        out[s].ut = P.ut;
        out[s].v = (dir == 1) ? P.ux : (dir == 2) ? P.uy : P.un;
        out[s].y = 1.0 / P.ut;
    }
}

/* --------------------------------------------------- bulk viscosity */
struct Zeta { int law; double norm, T0, w; };

/* SourceTerms.cpp:40-48 (T in fm^-1) or a Gaussian in T [GeV] */
__device__ __forceinline__ double zeta_over_s(const Zeta &Z, double T)
{
    if (Z.law == 1) {
        double z = (T * 0.197326938 - Z.T0) / Z.w;
        return Z.norm * exp(-(z * z));
    }
    double x = T / 1.01355;
    if (x > 1.05) return 0.9 * exp(-(x - 1) / 0.025) + 0.25 * exp(-(x - 1) / 0.13) + 0.001;
    else if (x < 0.995) return 0.9 * exp((x - 1) / 0.0025) + 0.22 * exp((x - 1) / 0.022) + 0.03;
    return -13.77 * x * x + 27.55 * x - 13.45;
}

/* a / b with y = RN(1/b): exact (div_rcp) in FP64, a * y in FP32 */
__device__ __forceinline__ double dvr(double a, double b, double y) { return div_rcp(a, b, y); }
__device__ __forceinline__ float dvr(float a, float, float y) { return a * y; }

/* How a body takes its quotients: PlainQuot each by itself (div_rcp and the
 * compiler's division in FP64, a * y in FP32); DirectQuot branch-free
 * (div_rn, rcp_rn), collecting the range tests: when fine() is false at the
 * end, or a result is not finite, the caller runs the body again with
 * PlainQuot.  DirectQuot's divisors are positive (lengths, times, u^tau). */
struct PlainQuot {
    template <typename R>
    __device__ __forceinline__ R operator()(R a, R b, R y) const { return dvr(a, b, y); }
    template <typename R>
    __device__ __forceinline__ R over(R a, R b) const { return a / b; }
    template <typename R>
    __device__ __forceinline__ R over_const(R a, R b, R) const { return a / b; }
    /* as operator() where the divisor's reciprocal pays only in the other form */
    template <typename R>
    __device__ __forceinline__ R quotient(R a, R b, R) const { return a / b; }
    __device__ __forceinline__ float root(float x) const { return sqrtf(x); }
    template <typename R>
    __device__ __forceinline__ R rcp(R b) const { return R(1.0) / b; }
    __device__ __forceinline__ double deriv(double th, double x, double y, double z) const { return approx_deriv(th, x, y, z); }
};
template <bool MIXED = false>
struct DirectQuot {
    unsigned key = ~0u;
    bool ok = true;
    __device__ __forceinline__ double operator()(double a, double b, double y)
    {
        key = min(key, div_key(a));
        return div_rn(a, b, y);
    }
    __device__ __forceinline__ double rcp(double b)
    {
        ok = ok && in_range(b) && rcp_ok(b);
        return rcp_rn(b);
    }
    __device__ __forceinline__ double over(double a, double b) { return (*this)(a, b, rcp(b)); }
    __device__ __forceinline__ double over_const(double a, double b, double y) { return (*this)(a, b, y); }
    __device__ __forceinline__ double quotient(double a, double b, double y) { return (*this)(a, b, y); }
    __device__ __forceinline__ float root(float x)
    {
        ok = ok && in_range(x);
        return root32<MIXED>(x);
    }
    __device__ __forceinline__ double deriv(double th, double x, double y, double z) const { return limited(th, x, y, z, 0x3ff00000); }
    __device__ __forceinline__ bool fine() const { return ok && key >= kDivKeyLo; }
};

/* the temperature and, where a^2 = (1/3 - cs^2)^2 vanishes, the bulk
 * relaxation rate 15 a^2 T / (zeta/s), which is +0 whenever zeta/s > 0: the
 * exponential and the division are then left out (the Gaussian law is
 * positive while its exponent stays clear of underflow, the reference's law
 * everywhere) */
template <int EOS>
__device__ __forceinline__ double temperature(PlainQuot &, const DevEos &E, double e) { return eos_T<EOS>(E, e); }
template <int EOS>
__device__ __forceinline__ double temperature(DirectQuot<> &dv, const DevEos &E, double e)
{
    dv.ok = dv.ok && in_range(e);
    if (EOS == 1) return floor15(eos_interp_direct(E, e, E.T_tb));
    return (double)powf_quarter(__double2float_rn(dv.over(e, E.a)), E.pq);
}
__device__ __forceinline__ double bulk_rate(PlainQuot &, const Zeta &Z, double a2, double T) { return 15 * a2 * T / zeta_over_s(Z, T); }
__device__ __forceinline__ double bulk_rate(DirectQuot<> &dv, const Zeta &Z, double a2, double T)
{
    const double z = (T * 0.197326938 - Z.T0) / Z.w;
    const bool positive = Z.law != 1 || (Z.norm >= 0x1p-100 && z * z < 600.0);
    if (a2 == 0.0 && T > 0.0 && T < 0x1p100 && positive) return 0.0;
    return 15 * a2 * T / zeta_over_s(Z, T);
}

/* SourceTerms.cpp:55-313, the right-hand side of the pi^{mu nu} (and Pi)
 * relaxation equations divided by u^tau.  yt = RN(1/t); every division by
 * t, 2t, t^2 and 5 goes through the shared reciprocal (dvr: the same
 * quotient in FP64, a product in FP32). */
template <typename R, int EOS, bool BULK, class Quot>
__device__ __forceinline__ void pimunu_rhs(Quot &dv, const DevEos &E, const Zeta &Z, R *rhs, R t, R yt, double e_d, double p_d,
    double ut_d, double ux_d, double uy_d, double un_d, double utp, double uxp, double uyp, double unp,
    const R *pv, R Pi,
    R dxut, R dyut, R dnut, R dxux, R dyux, R dnux,
    R dxuy, R dyuy, R dnuy, R dxun, R dyun, R dnun, R dkvk,
    R d_etabar, R d_dt)
{
    const R ut = R(ut_d), ux = R(ux_d), uy = R(uy_d), un = R(un_d), e = R(e_d), p = R(p_d);
    const R delta_pipi = R(1.33333), tau_pipi = R(1.42857), delta_PiPi = R(0.666667), lambda_piPi = R(1.2);
    const R pitt = pv[0], pitx = pv[1], pity = pv[2], pitn = pv[3], pixx = pv[4];
    const R pixy = pv[5], pixn = pv[6], piyy = pv[7], piyn = pv[8], pinn = pv[9];
    R T = R(temperature<EOS>(dv, E, e_d));
    R taupiInv = dv.over(dv.over_const(T, R(5), R(0.2)), d_etabar);
    R beta_pi = dv(e + p, R(5), R(0.2));
    R cs2 = R(eos_cs2<EOS>(E, e_d));
    R a = R(1.0) / R(3.0) - cs2;
    R a2 = a * a;
    R beta_Pi = 15 * a2 * (e + p);
    R lambda_Pipi = dv(8 * a, R(5), R(0.2));
    R tauPiInv = R(0.0);
    /* in FP64 for both precisions: zeta/s underflows FP32 far from its peak
     * while a2 = 0 for both EoS kinds, and 0/0 must not appear */
    if (BULK) tauPiInv = R(bulk_rate(dv, Z, double(a2), double(T)));
    R ut2 = ut * ut, un2 = un * un, t2 = t * t, t3 = t * t2;
    const R yt2 = dv.rcp(t2), y2t = yt * R(0.5);   /* RN(1/t^2); RN(1/(2t)) = RN(1/t) / 2 */
    const R kThird = R(1.0) / R(3.0), yut = dv.rcp(ut), ydt = dv.rcp(d_dt);
    R dtut = dv(R(ut_d - utp), d_dt, ydt), dtux = dv(R(ux_d - uxp), d_dt, ydt), dtuy = dv(R(uy_d - uyp), d_dt, ydt), dtun = dv(R(un_d - unp), d_dt, ydt);
    R Dut = ut * dtut + ux * dxut + uy * dyut + un * dnut + t * un * un;
    R DuxUpper = ut * dtux + ux * dxux + uy * dyux + un * dnux;
    R Dux = -DuxUpper;
    R DuyUpper = ut * dtuy + ux * dxuy + uy * dyuy + un * dnuy;
    R Duy = -DuyUpper;
    R DunUpper = ut * dtun + ux * dxun + uy * dyun + un * dnun + dv(2 * ut * un, t, yt);
    R Dun = -t2 * DunUpper;
    R dut = Dut - t * un * un;
    R dux = ut * dtux + ux * dxux + uy * dyux + un * dnux;
    R duy = ut * dtuy + ux * dxuy + uy * dyuy + un * dnuy;
    R dun = ut * dtun + ux * dxun + uy * dyun + un * dnun;
    R theta = dv(ut, t, yt) + dtut + dxux + dyuy + dnun;
    R stt = -t * ut * un2 + (dtut - ut * dut) + dv((ut2 - 1) * theta, R(3.0), kThird);
    R stx = -(t * un2 * ux) / R(2.0) + (dtux - dxut) / R(2.0) - (ux * dut + ut * dux) / R(2.0) + dv(ut * ux * theta, R(3.0), kThird);
    R sty = -(t * un2 * uy) / R(2.0) + (dtuy - dyut) / R(2.0) - (uy * dut + ut * duy) / R(2.0) + dv(ut * uy * theta, R(3.0), kThird);
    R stn = dv(-un * (R(2.0) * ut2 + t2 * un2), R(2.0) * t, y2t) + (dtun - dv(dnut, t2, yt2)) / R(2.0) - (un * dut + ut * dun) / R(2.0) + dv(ut * un * theta, R(3.0), kThird);
    R sxx = -(dxux + ux * dux) + dv((R(1.0) + ux * ux) * theta, R(3.0), kThird);
    R sxy = -(dxuy + dyux) / R(2.0) - (uy * dux + ux * duy) / R(2.0) + dv(ux * uy * theta, R(3.0), kThird);
    R sxn = dv(-ut * ux * un, t, yt) - (dxun + dv(dnux, t2, yt2)) / R(2.0) - (un * dux + ux * dun) / R(2.0) + dv(ux * un * theta, R(3.0), kThird);
    R syy = -(dyuy + uy * duy) + dv((R(1.0) + uy * uy) * theta, R(3.0), kThird);
    R syn = dv(-ut * uy * un, t, yt) - (dyun + dv(dnuy, t2, yt2)) / R(2.0) - (un * duy + uy * dun) / R(2.0) + dv(uy * un * theta, R(3.0), kThird);
    R snn = dv.over(-ut * (R(1.0) + R(2.0) * t2 * un2), t3) - dv(dnun, t2, yt2) - un * dun + dv((yt2 + un2) * theta, R(3.0), kThird);
    R wtx = (-dtux - dxut + ut * dux - ux * dut - t * un2 * ux) / R(2.0);
    R wty = (-dtuy - dyut + ut * duy - uy * dut - t * un2 * uy) / R(2.0);
    R wtn = (-t2 * dtun - R(2.0) * t * un - dnut - ut * Dun - t2 * un * dut - t3 * un * un2) / R(2.0);
    R wxy = (dxuy - dyux + ux * duy - uy * dux) / R(2.0);
    R wxn = (t2 * dxun - dnux - ux * Dun - t2 * un * dux) / R(2.0);
    R wyn = (t2 * dyun - dnuy - uy * Dun - t2 * un * duy) / R(2.0);
    R wxt = wtx, wyt = wty, wnt = dv(wtn, t2, yt2), wyx = -wxy, wnx = dv(-wxn, t2, yt2), wny = dv(-wyn, t2, yt2);
    R I1tt = R(2.0) * ut * (pitt * Dut + pitx * Dux + pity * Duy + pitn * Dun);
    R I1tx = (pitt * ux + pitx * ut) * Dut + (pitx * ux + pixx * ut) * Dux + (pity * ux + pixy * ut) * Duy + (pitn * ux + pixn * ut) * Dun;
    R I1ty = (pitt * uy + pity * ut) * Dut + (pitx * uy + pixy * ut) * Dux + (pity * uy + piyy * ut) * Duy + (pitn * uy + piyn * ut) * Dun;
    R I1tn = (pitt * un + pitn * ut) * Dut + (pitx * un + pixn * ut) * Dux + (pity * un + piyn * ut) * Duy + (pitn * un + pinn * ut) * Dun;
    R I1xx = R(2.0) * ux * (pitx * Dut + pixx * Dux + pixy * Duy + pixn * Dun);
    R I1xy = (pitx * uy + pity * ux) * Dut + (pixx * uy + pixy * ux) * Dux + (pixy * uy + piyy * ux) * Duy + (pixn * uy + piyn * ux) * Dun;
    R I1xn = (pitx * un + pitn * ux) * Dut + (pixx * un + pixn * ux) * Dux + (pixy * un + piyn * ux) * Duy + (pixn * un + pinn * ux) * Dun;
    R I1yy = R(2.0) * uy * (pity * Dut + pixy * Dux + piyy * Duy + piyn * Dun);
    R I1yn = (pity * un + pitn * uy) * Dut + (pixy * un + pixn * uy) * Dux + (piyy * un + piyn * uy) * Duy + (piyn * un + pinn * uy) * Dun;
    R I1nn = R(2.0) * un * (pitn * Dut + pixn * Dux + piyn * Duy + pinn * Dun);
    R I2tt = theta * pitt, I2tx = theta * pitx, I2ty = theta * pity, I2tn = theta * pitn, I2xx = theta * pixx;
    R I2xy = theta * pixy, I2xn = theta * pixn, I2yy = theta * piyy, I2yn = theta * piyn, I2nn = theta * pinn;
    R I3tt = R(2.0) * (pitx * wtx + pity * wty + pitn * wtn);
    R I3tx = pitt * wxt + pity * wxy + pitn * wxn + pixx * wtx + pixy * wty + pixn * wtn;
    R I3ty = pitt * wyt + pitx * wyx + pitn * wyn + pixy * wtx + piyy * wty + piyn * wtn;
    R I3tn = pitt * wnt + pitx * wnx + pity * wny + pixn * wtx + piyn * wty + pinn * wtn;
    R I3xx = R(2.0) * (pitx * wxt + pixy * wxy + pixn * wxn);
    R I3xy = pitx * wyt + pity * wxt + pixx * wyx + piyy * wxy + pixn * wyn + piyn * wxn;
    R I3xn = pitx * wnt + pitn * wxt + pixx * wnx + pixy * wny + piyn * wxy + pinn * wxn;
    R I3yy = R(2.0) * (pity * wyt + pixy * wyx + piyn * wyn);
    R I3yn = pity * wnt + pitn * wyt + pixy * wnx + pixn * wyx + piyy * wny + pinn * wyn;
    R I3nn = R(2.0) * (pitn * wnt + pixn * wnx + piyn * wny);
    R ux2 = ux * ux, uy2 = uy * uy;
    R ps = pitt * stt - R(2.0) * pitx * stx - R(2.0) * pity * sty + pixx * sxx + R(2.0) * pixy * sxy + piyy * syy - R(2.0) * pitn * stn * t2 + R(2.0) * pixn * sxn * t2 + R(2.0) * piyn * syn * t2 + pinn * snn * t2 * t2;
    R I4tt = (pitt * stt - pitx * stx - pity * sty - t2 * pitn * stn) - dv((R(1.0) - ut2) * ps, R(3.0), kThird);
    R I4tx = (pitt * stx + pitx * stt) / R(2.0) - (pitx * sxx + pixx * stx) / R(2.0) - (pity * sxy + pixy * sty) / R(2.0) - t2 * (pitn * sxn + pixn * stn) / R(2.0) + dv((ut * ux) * ps, R(3.0), kThird);
    R I4ty = (pitt * sty + pity * stt) / R(2.0) - (pitx * sxy + pixy * stx) / R(2.0) - (pity * syy + piyy * sty) / R(2.0) - t2 * (pitn * syn + piyn * stn) / R(2.0) + dv((ut * uy) * ps, R(3.0), kThird);
    R I4tn = (pitt * stn + pitn * stt) / R(2.0) - (pitx * sxn + pixn * stx) / R(2.0) - (pity * syn + piyn * sty) / R(2.0) - t2 * (pitn * snn + pinn * stn) / R(2.0) + dv((ut * un) * ps, R(3.0), kThird);
    R I4xx = (pitx * stx - pixx * sxx - pixy * sxy - t2 * pixn * sxn) + dv((R(1.0) + ux2) * ps, R(3.0), kThird);
    R I4xy = (pitx * sty + pity * stx) / R(2.0) - (pixx * sxy + pixy * sxx) / R(2.0) - (pixy * syy + piyy * sxy) / R(2.0) - t2 * (pixn * syn + piyn * sxn) / R(2.0) + dv((ux * uy) * ps, R(3.0), kThird);
    R I4xn = (pitx * stn + pitn * stx) / R(2.0) - (pixx * sxn + pixn * sxx) / R(2.0) - (pixy * syn + piyn * sxy) / R(2.0) - t2 * (pixn * snn + pinn * sxn) / R(2.0) + dv((ux * un) * ps, R(3.0), kThird);
    R I4yy = (pity * sty - pixy * sxy - piyy * syy - t2 * piyn * syn) + dv((R(1.0) + uy2) * ps, R(3.0), kThird);
    R I4yn = (pity * stn + pitn * sty) / R(2.0) - (pixy * sxn + pixn * sxy) / R(2.0) - (piyy * syn + piyn * syy) / R(2.0) - t2 * (piyn * snn + pinn * syn) / R(2.0) + dv((uy * un) * ps, R(3.0), kThird);
    R I4nn = (pitn * stn - pixn * sxn - piyn * syn - t2 * pinn * snn) + dv((yt2 + un2) * ps, R(3.0), kThird);
    R Itt = I1tt + delta_pipi * I2tt - I3tt + tau_pipi * I4tt - lambda_piPi * Pi * stt;
    R Itx = I1tx + delta_pipi * I2tx - I3tx + tau_pipi * I4tx - lambda_piPi * Pi * stx;
    R Ity = I1ty + delta_pipi * I2ty - I3ty + tau_pipi * I4ty - lambda_piPi * Pi * sty;
    R Itn = I1tn + delta_pipi * I2tn - I3tn + tau_pipi * I4tn - lambda_piPi * Pi * stn;
    R Ixx = I1xx + delta_pipi * I2xx - I3xx + tau_pipi * I4xx - lambda_piPi * Pi * sxx;
    R Ixy = I1xy + delta_pipi * I2xy - I3xy + tau_pipi * I4xy - lambda_piPi * Pi * sxy;
    R Ixn = I1xn + delta_pipi * I2xn - I3xn + tau_pipi * I4xn - lambda_piPi * Pi * sxn;
    R Iyy = I1yy + delta_pipi * I2yy - I3yy + tau_pipi * I4yy - lambda_piPi * Pi * syy;
    R Iyn = I1yn + delta_pipi * I2yn - I3yn + tau_pipi * I4yn - lambda_piPi * Pi * syn;
    R Inn = I1nn + delta_pipi * I2nn - I3nn + tau_pipi * I4nn - lambda_piPi * Pi * snn;
    R dpitt = R(2.0) * beta_pi * stt - pitt * taupiInv - Itt - R(2.0) * un * t * pitn;
    R dpitx = R(2.0) * beta_pi * stx - pitx * taupiInv - Itx - un * t * pixn;
    R dpity = R(2.0) * beta_pi * sty - pity * taupiInv - Ity - un * t * piyn;
    R dpitn = R(2.0) * beta_pi * stn - pitn * taupiInv - Itn - un * t * pinn - dv(ut * pitn + un * pitt, t, yt);
    R dpixx = R(2.0) * beta_pi * sxx - pixx * taupiInv - Ixx;
    R dpixy = R(2.0) * beta_pi * sxy - pixy * taupiInv - Ixy;
    R dpixn = R(2.0) * beta_pi * sxn - pixn * taupiInv - Ixn - dv(ut * pixn + un * pitx, t, yt);
    R dpiyy = R(2.0) * beta_pi * syy - piyy * taupiInv - Iyy;
    R dpiyn = R(2.0) * beta_pi * syn - piyn * taupiInv - Iyn - dv(ut * piyn + un * pity, t, yt);
    R dpinn = R(2.0) * beta_pi * snn - pinn * taupiInv - Inn - dv(2 * (ut * pinn + un * pitn), t, yt);
    rhs[0] = dv(dpitt, ut, yut) + pitt * dkvk;
    rhs[1] = dv(dpitx, ut, yut) + pitx * dkvk;
    rhs[2] = dv(dpity, ut, yut) + pity * dkvk;
    rhs[3] = dv(dpitn, ut, yut) + pitn * dkvk;
    rhs[4] = dv(dpixx, ut, yut) + pixx * dkvk;
    rhs[5] = dv(dpixy, ut, yut) + pixy * dkvk;
    rhs[6] = dv(dpixn, ut, yut) + pixn * dkvk;
    rhs[7] = dv(dpiyy, ut, yut) + piyy * dkvk;
    rhs[8] = dv(dpiyn, ut, yut) + piyn * dkvk;
    rhs[9] = dv(dpinn, ut, yut) + pinn * dkvk;
    if (BULK) {
        R dPi = -beta_Pi * theta - Pi * tauPiInv - delta_PiPi * Pi * theta + lambda_Pipi * ps;
        rhs[10] = dv(dPi, ut, yut) + Pi * dkvk;
    }
}

} // namespace vh

#endif
