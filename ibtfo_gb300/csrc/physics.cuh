// Device-side physics of the IBTFO update: limiters, physical fluxes and the
// three Riemann solvers, written so that every expression is evaluated in
// the same order as the reference (the parity build compiles with
// -fmad=false, so no multiply-add is fused and each result is the IEEE
// binary64 value of the reference expression).
//
// pow(x, 0.5) of the reference is evaluated as a correctly rounded square
// root; both agree except where the library pow is off by its last bit.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "int64math.cuh"
#include "internal.h"

namespace ibtfo {

enum Scheme { MUSCL = 0, MHM = 1, GODUNOV = 2, LAX = 3 };
enum Riemann { HLL = 0, HLLC = 1, PVRS = 2, SW = 3, HLLCT = 4, HLLT = 5 };
// the solver keys with no reference counterpart that carry the positivity
// safeguards (first-order fallback of unphysical face pairs, pressure floor)
constexpr bool safeguarded(int rie) { return rie == HLLCT || rie == HLLT; }
enum Limiter { MINMOD = 0, VANLEER = 1 };

// x >= 0 and x <= 0 as IEEE comparisons give them (false for NaN), on the integer pipe
__device__ __forceinline__ bool ge0(double x)
{
    const long long b = __double_as_longlong(x);
    return (b >= 0 && b <= 0x7ff0000000000000LL) || b == (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool le0(double x)
{
    const long long b = __double_as_longlong(x);
    return b == 0 || (b < 0 && b <= (long long)0xfff0000000000000ULL);
}

// The bits of |x|, masked on the high word: masking a double's 64 bits at
// once is taken for fabs, which is an FP64 addition on this part (12 of a
// face's 24 additions, before).
__device__ __forceinline__ long long magnitude_bits(double x)
{
    return ((long long)(__double2hiint(x) & 0x7fffffff) << 32) | (unsigned)__double2loint(x);
}
__device__ __forceinline__ double magnitude(double x)
{
    return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}

// pow(x, 0.5): +0 for a zero of either sign (as pow gives), sqrt otherwise
__device__ __forceinline__ double pow_half(double x)
{
    return (__double_as_longlong(x) << 1) == 0 ? 0.0 : sqrt_rn(x);
}

// Src/Base/Slope_limiter/minmod/Slope_limiter.H:4:
//   ((a*b) > 0) ? ((a/b > 1) ? b : a) : 0
// evaluated on the integer pipe with the same result:
// * a*b > 0 holds when a and b are non-zero, not NaN, of the same sign, and
//   the product does not underflow to zero; for biased exponents
//   ea + eb >= 972 (both normal) |a*b| >= 2^-1074 cannot underflow, below
//   that the product itself is evaluated;
// * where a*b > 0, the rounded quotient a/b exceeds 1 exactly when |a| > |b|:
//   for doubles |a| > |b| implies |a|/|b| >= 1 + ulp(b)/|b| > 1 + 2^-53,
//   which rounds above 1, and |a| <= |b| gives a quotient <= 1; magnitudes of
//   non-NaN doubles order like their bit patterns.
static __device__ __noinline__ bool product_positive(double a, double b) { return (a * b) > 0; }
__device__ __forceinline__ double lim_minmod(double a, double b)
{
    const long long ma = magnitude_bits(a), mb = magnitude_bits(b);
    bool pos = ((__double2hiint(a) ^ __double2hiint(b)) >= 0) && ma != 0 && mb != 0 && ma <= 0x7ff0000000000000LL &&
               mb <= 0x7ff0000000000000LL;
    if (pos)
    {
        const int ea = (int)(ma >> 52), eb = (int)(mb >> 52);
        if (!(ea != 0 && eb != 0 && ea + eb >= 972))
            pos = product_positive(a, b);
    }
    return pos ? ((ma > mb) ? b : a) : 0.0;
}

// Src/Base/Slope_limiter/VanLeer/Slope_limiter.H:4 as the macro expands at its
// call sites, where b is the text `P - Q`: (r*r + r) * P - Q / (r*r + 1)
__device__ __forceinline__ double lim_vanleer(double a, double P, double Q)
{
    double b = P - Q;
    double r = divide_rn(a + 1e-7, divisor(b + 1e-7));
    return (r > 0) ? ((r * r + r) * P - divide_rn(Q, divisor(r * r + 1))) : 0.0;
}

// limiter(hi - lo, P - Q), and half of it
template <int LIM>
__device__ __forceinline__ double limited(double hi, double lo, double P, double Q)
{
    if (LIM == VANLEER)
        return lim_vanleer(hi - lo, P, Q);
    return lim_minmod(hi - lo, P - Q);
}
template <int LIM>
__device__ __forceinline__ double half_slope(double hi, double lo, double P, double Q)
{
    return 0.5 * limited<LIM>(hi, lo, P, Q);
}

// Face states of one interface from the four cells c0..c3 along the sweep
// (interface between c1 and c2).  MUSCL_Scheme.cpp:39-41 and :55-57 (and the
// Y forms :100-102, :116-118): U_L = c1 + 0.5 lim(c1-c0, c2-c1),
// U_R = c2 - 0.5 lim(c3-c2, c2-c1).  Godunov: U_L = c1, U_R = c2.
template <int SCH, int LIM>
__device__ __forceinline__ void face_states(const double c0[4], const double c1[4], const double c2[4],
                                            const double c3[4], double UL[4], double UR[4])
{
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
        if (SCH == GODUNOV)
        {
            UL[k] = c1[k];
            UR[k] = c2[k];
        }
        else
        {
            // c +- RN(0.5 s): halving is exact, so one fused operation rounds as the two do
            UL[k] = fma(0.5, limited<LIM>(c1[k], c0[k], c2[k], c1[k]), c1[k]);
            UR[k] = fma(-0.5, limited<LIM>(c3[k], c2[k], c2[k], c1[k]), c2[k]);
        }
    }
}

// Conserve2FluxX (Src/Base/Common/Conserve2Flux.cpp:66-74)
__device__ __forceinline__ void flux_x(const double U[4], double g, double F[4])
{
    double rho = U[0];
    double u = U[1] / rho;
    double v = U[2] / rho;
    double p = (g - 1) * (U[3] - 0.5 * rho * (u * u + v * v));
    F[0] = rho * u;
    F[1] = rho * u * u + p;
    F[2] = rho * u * v;
    F[3] = (U[3] + p) * u;
}

// Conserve2FluxY (Src/Base/Common/Conserve2Flux.cpp:101-109)
__device__ __forceinline__ void flux_y(const double U[4], double g, double G[4])
{
    double rho = U[0];
    double u = U[1] / rho;
    double v = U[2] / rho;
    double p = (g - 1) * (U[3] - 0.5 * rho * (u * u + v * v));
    G[0] = rho * v;
    G[1] = rho * u * v;
    G[2] = rho * v * v + p;
    G[3] = (U[3] + p) * v;
}

// The states of a face as the strict solvers use them: every quotient by rho
// shares one reciprocal (divide_rn gives the IEEE quotient).  Conserve2FluxX /
// Conserve2FluxY (Conserve2Flux.cpp:66-74, :101-109) evaluated from them.
struct StrictPrim
{
    double rho, u, v, p, E;
    Divisor by_rho;
};
__device__ __forceinline__ StrictPrim strict_prim(const double U[4], const GridDesc &g)
{
    StrictPrim s;
    s.rho = U[0];
    s.by_rho = divisor(U[0]);
    s.u = divide_rn(U[1], s.by_rho);
    s.v = divide_rn(U[2], s.by_rho);
    s.E = U[3];
    s.p = g.gm1 * (U[3] - 0.5 * s.rho * (s.u * s.u + s.v * s.v));
    return s;
}
template <int NRM>
__device__ __forceinline__ void strict_flux(const StrictPrim &s, double F[4])
{
    const double q = (NRM == 1) ? s.u : s.v;
    F[0] = s.rho * q;
    F[NRM] = s.rho * q * q + s.p;
    F[3 - NRM] = s.rho * s.u * s.v;
    F[3] = (s.E + s.p) * q;
}

// MHM half-step predictor on the two states of one interface,
// MHM_Scheme.cpp:73-93 (X, h = dx) and :160-180 (Y, h = dy):
// U += 0.5 * (F(U_L) - F(U_R)) * dt / h for both states (the halving commutes
// with the roundings that follow it).
template <int NRM>
__device__ __forceinline__ void mhm_predict(double UL[4], double UR[4], const GridDesc &g, double dt)
{
    const Divisor &by_h = (NRM == 1) ? g.by_dx : g.by_dy;
    double FL[4], FR[4];
    strict_flux<NRM>(strict_prim(UL, g), FL);
    strict_flux<NRM>(strict_prim(UR, g), FR);
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
        const double q = divide_rn((FL[k] - FR[k]) * dt, by_h);
        UL[k] = fma(0.5, q, UL[k]);
        UR[k] = fma(0.5, q, UR[k]);
    }
}

// ----------------------------------------------------------------- HLL

// HLL/Riemann_solver.cpp:131-169 (X), :202-235 (Y).  Y: returns false when
// S_D >= 0 (the reference then stores nothing and the slot keeps the X-face
// flux, :224-227).  The reference's halvings are exact and are moved past the
// roundings they commute with:
//   p_star = 0.5 (p_L + p_R) + 0.5 (u_L - u_R) (0.5 (rho_L + rho_R) 0.5 (a_L + a_R)),
//   (g + 1) p_star / 2 / g / p_K + (g - 1) / 2 / g
template <int NRM>
__device__ __forceinline__ bool strict_hll(const double UL[4], const double UR[4], const GridDesc &g, double F[4])
{
    const StrictPrim L = strict_prim(UL, g), R = strict_prim(UR, g);
    const double qL = (NRM == 1) ? L.u : L.v, qR = (NRM == 1) ? R.u : R.v;
    const double aL = pow_half(divide_rn(g.gamma * L.p, L.by_rho));
    const double aR = pow_half(divide_rn(g.gamma * R.p, R.by_rho));
    const double z = (qL - qR) * ((L.rho + R.rho) * (aL + aR));
    const double p_star = fma(0.125, z, 0.5 * (L.p + R.p));
    const double t = divide_rn(g.gp1 * p_star, g.by_g);
    const double S_L = qL - aL * sqrt_rn(fma(0.5, divide_rn(t, divisor(L.p)), g.hgm1g));
    if (NRM == 2 && ge0(S_L))
        return false;
    const double S_R = qR + aR * sqrt_rn(fma(0.5, divide_rn(t, divisor(R.p)), g.hgm1g));
    if (ge0(S_L))
        strict_flux<NRM>(L, F);
    else if (le0(S_R))
        strict_flux<NRM>(R, F);
    else
    {
        double FL[4], FR[4];
        strict_flux<NRM>(L, FL);
        strict_flux<NRM>(R, FR);
        const Divisor by_w = divisor(S_R - S_L);
        const double SS = S_R * S_L;
#pragma unroll
        for (int k = 0; k < 4; k++)
            F[k] = divide_rn(S_R * FL[k] - S_L * FR[k] + SS * (UR[k] - UL[k]), by_w);
    }
    return true;
}

// ----------------------------------------------------------------- PVRS

// PVRS/Riemann_solver.cpp:308-435 (X), with the reference's S_TL/S_TR (both use
// p_star/p_R, :331,:334) and fan states (rho in place of u, :375-377).
__device__ __forceinline__ void pvrs_x(const double UL[4], const double UR[4], double g, double F[4])
{
    double rho_L = UL[0], rho_R = UR[0];
    double u_L = UL[1] / rho_L;
    double v_L = UL[2] / rho_L;
    double p_L = (g - 1) * (UL[3] - 0.5 * rho_L * (u_L * u_L + v_L * v_L));
    double u_R = UR[1] / rho_R;
    double v_R = UR[2] / rho_R;
    double p_R = (g - 1) * (UR[3] - 0.5 * rho_R * (u_R * u_R + v_R * v_R));
    double a_L = pow_half(g * p_L / rho_L);
    double a_R = pow_half(g * p_R / rho_R);
    double rho_bar = 0.5 * (rho_L + rho_R);
    double a_bar = 0.5 * (a_L + a_R);
    double p_star = 0.5 * (p_L + p_R) + 0.5 * (u_L - u_R) * (rho_bar * a_bar);
    double u_star = 0.5 * (u_L + u_R) + 0.5 * (p_L - p_R) / (rho_bar * a_bar);
    double rhoL_star = rho_L + (p_star - p_L) / a_L / a_L;
    double rhoR_star = rho_R + (p_star - p_R) / a_R / a_R;
    double S_L = u_L - a_L * sqrt((g + 1) * p_star / 2 / g / p_L + (g - 1) / 2 / g);
    double S_R = u_R + a_R * sqrt((g + 1) * p_star / 2 / g / p_R + (g - 1) / 2 / g);
    double S_HL = u_L - a_L;
    double S_TL = u_star - pow(a_L * (p_star / p_R), ((g - 1) / 2 / g));
    double S_HR = u_R + a_R;
    double S_TR = u_star + pow(a_R * (p_star / p_R), ((g - 1) / 2 / g));
    // 0: left direct, 1: left star, 2: left fan, 3: right direct, 4: right star, 5: right fan
    int br;
    if (u_star > 0)
    {
        if (p_star > p_L)
            br = (S_L > 0) ? 0 : 1;
        else
            br = (S_HL > 0) ? 0 : ((S_TL < 0) ? 1 : 2);
    }
    else
    {
        if (p_star > p_R)
            br = (S_R < 0) ? 3 : 4;
        else
            br = (S_HR < 0) ? 3 : ((S_TR > 0) ? 4 : 5);
    }
    if (br == 0)
    {
        F[0] = rho_L * u_L;
        F[1] = rho_L * u_L * u_L + p_L;
        F[2] = rho_L * u_L * v_L;
        F[3] = (UL[3] + p_L) * u_L;
    }
    else if (br == 3)
    {
        F[0] = rho_R * u_R;
        F[1] = rho_R * u_R * u_R + p_R;
        F[2] = rho_R * u_R * v_R;
        F[3] = (UR[3] + p_R) * u_R;
    }
    else if (br == 1 || br == 4)
    {
        double rs = (br == 1) ? rhoL_star : rhoR_star;
        double vt = (br == 1) ? v_L : v_R;
        F[0] = rs * u_star;
        F[1] = rs * u_star * u_star + p_star;
        F[2] = rs * u_star * vt;
        F[3] = (g * p_star / (g - 1) + 0.5 * rs * (u_star * u_star + vt * vt)) * u_star;
    }
    else
    {
        double rho_s = (br == 2) ? rho_L : rho_R;
        double a_s = (br == 2) ? a_L : a_R;
        double u_s = (br == 2) ? u_L : u_R;
        double p_s = (br == 2) ? p_L : p_R;
        double vt = (br == 2) ? v_L : v_R;
        double rho_f = rho_s * pow(2 / (g + 1) + (g - 1) * (rho_s) / (g + 1) / a_s, 2 / (g - 1));
        double u_f = 2 * (a_s + (g - 1) * u_s / 2) / (g + 1);
        double p_f = p_s * pow((2 / (g + 1) + (g - 1) * (rho_s) / (g + 1) / a_s), 2 * g / (g - 1));
        F[0] = rho_f * u_f;
        F[1] = rho_f * u_f * u_f + p_f;
        F[2] = rho_f * u_f * vt;
        F[3] = (g * p_f / (g - 1) + 0.5 * rho_f * (u_f * u_f + vt * vt)) * u_f;
    }
}

// PVRS/Riemann_solver.cpp:463-590 (Y).  Returns a mask of components the
// reference leaves unchanged in the shared flux slot: the branch at :547-550
// stores its energy flux elsewhere, so component 3 keeps the X-face flux.
// *stray receives that energy flux when the branch fires.
__device__ __forceinline__ int pvrs_y(const double UD[4], const double UU[4], double g, double G[4], double *stray)
{
    double rho_U = UU[0], rho_D = UD[0];
    double u_U = UU[1] / rho_U;
    double v_U = UU[2] / rho_U;
    double p_U = (g - 1) * (UU[3] - 0.5 * rho_U * (u_U * u_U + v_U * v_U));
    double u_D = UD[1] / rho_D;
    double v_D = UD[2] / rho_D;
    double p_D = (g - 1) * (UD[3] - 0.5 * rho_D * (u_D * u_D + v_D * v_D));
    double a_U = pow_half(g * p_U / rho_U);
    double a_D = pow_half(g * p_D / rho_D);
    double rho_bar = 0.5 * (rho_U + rho_D);
    double a_bar = 0.5 * (a_U + a_D);
    double p_star = 0.5 * (p_U + p_D) + 0.5 * (v_D - v_U) * (rho_bar * a_bar);
    double v_star = 0.5 * (v_D + v_U) + 0.5 * (p_D - p_U) / (rho_bar * a_bar);
    double rhoD_star = rho_D + (p_star - p_D) / a_D / a_D;
    double rhoU_star = rho_U + (p_star - p_U) / a_U / a_U;
    double S_D = v_D - a_D * sqrt((g + 1) * p_star / 2 / g / p_D + (g - 1) / 2 / g);
    double S_U = v_U + a_U * sqrt((g + 1) * p_star / 2 / g / p_U + (g - 1) / 2 / g);
    double S_HD = v_D - a_D;
    double S_TD = v_star - pow(a_D * (p_star / p_U), ((g - 1) / 2 / g));
    double S_HU = v_U + a_U;
    double S_TU = v_star + pow(a_U * (p_star / p_U), ((g - 1) / 2 / g));
    // 0: down direct, 1: down star, 2: down fan, 3: up direct, 4: up star, 5: up fan, 6: up direct (:547-550)
    int br;
    if (v_star > 0)
    {
        if (p_star > p_D)
            br = (S_D > 0) ? 0 : 1;
        else
            br = (S_HD > 0) ? 0 : ((S_TD < 0) ? 1 : 2);
    }
    else
    {
        if (p_star > p_U)
            br = (S_U < 0) ? 6 : 4;
        else
            br = (S_HU < 0) ? 3 : ((S_TU > 0) ? 4 : 5);
    }
    int keep = 0;
    if (br == 0)
    {
        G[0] = rho_D * v_D;
        G[1] = rho_D * u_D * v_D;
        G[2] = rho_D * v_D * v_D + p_D;
        G[3] = (UD[3] + p_D) * v_D;
    }
    else if (br == 3 || br == 6)
    {
        G[0] = rho_U * v_U;
        G[1] = rho_U * u_U * v_U;
        G[2] = rho_U * v_U * v_U + p_U;
        G[3] = (UU[3] + p_U) * v_U;
        if (br == 6)
        {
            *stray = G[3];
            keep = 1 << 3;
        }
    }
    else if (br == 1 || br == 4)
    {
        double rs = (br == 1) ? rhoD_star : rhoU_star;
        double ut = (br == 1) ? u_D : u_U;
        G[0] = rs * v_star;
        G[1] = rs * v_star * ut;
        G[2] = rs * v_star * v_star + p_star;
        G[3] = (g * p_star / (g - 1) + 0.5 * rs * (v_star * v_star + ut * ut)) * v_star;
    }
    else
    {
        double rho_s = (br == 2) ? rho_D : rho_U;
        double a_s = (br == 2) ? a_D : a_U;
        double v_s = (br == 2) ? v_D : v_U;
        double p_s = (br == 2) ? p_D : p_U;
        double ut = (br == 2) ? u_D : u_U;
        double rho_f = rho_s * pow(2 / (g + 1) + (g - 1) * (rho_s) / (g + 1) / a_s, 2 / (g - 1));
        double v_f = 2 * (a_s + (g - 1) * v_s / 2) / (g + 1);
        double p_f = p_s * pow((2 / (g + 1) + (g - 1) * (rho_s) / (g + 1) / a_s), 2 * g / (g - 1));
        G[0] = rho_f * v_f;
        G[1] = rho_f * v_f * ut;
        G[2] = rho_f * v_f * v_f + p_f;
        G[3] = (g * p_f / (g - 1) + 0.5 * rho_f * (v_f * v_f + ut * ut)) * v_f;
    }
    return keep;
}

// ----------------------------------------------------------- Steger-Warming

// StegerWarming/Riemann_solver.cpp:173-234 (X), :262-325 (Y): F = F+(U_L) + F-(U_R).
// Halves (x / 2) are exact and move past the roundings they commute with.
template <int NRM, int SIGN>
__device__ __forceinline__ void strict_sw_split(const double U[4], const GridDesc &g, double f[4])
{
    const StrictPrim s = strict_prim(U, g);
    const double a = pow_half(divide_rn(g.gamma * s.p, s.by_rho));
    const double e = divide_rn(divide_rn(s.p, g.by_gm1), s.by_rho);
    const double h = fma(0.5, s.v * s.v, fma(0.5, s.u * s.u, e)) + divide_rn(s.p, s.by_rho);
    const double delta = 1e-6;
    auto lam = [&](double x) {
        const double r = sqrt_rn(x * x + delta * delta);
        return 0.5 * (SIGN > 0 ? x + r : x - r);
    };
    const double q = (NRM == 1) ? s.u : s.v, w = (NRM == 1) ? s.v : s.u;
    const double l1 = lam(q), l3 = lam(q - a), l4 = lam(q + a);
    f[0] = divide_rn(0.5 * (s.rho * (g.gm1x2 * l1 + l3 + l4)), g.by_g);
    f[NRM] = divide_rn(0.5 * (s.rho * (g.gm1x2 * q * l1 + (q - a) * l3 + (q + a) * l4)), g.by_g);
    f[3 - NRM] = divide_rn(0.5 * (s.rho * (g.gm1x2 * w * l1 + l3 * w + l4 * w)), g.by_g);
    f[3] = divide_rn(0.5 * (s.rho * (g.gm1 * (s.u * s.u + s.v * s.v) * l1 + (h - a * q) * l3 + (h + a * q) * l4)),
                     g.by_g);
}
template <int NRM>
__device__ __forceinline__ void strict_sw(const double UL[4], const double UR[4], const GridDesc &g, double F[4])
{
    double fp[4], fn[4];
    strict_sw_split<NRM, 1>(UL, g, fp);
    strict_sw_split<NRM, -1>(UR, g, fn);
#pragma unroll
    for (int k = 0; k < 4; k++)
        F[k] = fp[k] + fn[k];
}

// ---------------------------------------------------------------- PVRS stray store
//
// In the reference's PVRS Y solver the branch at PVRS/Riemann_solver.cpp:547-550
// stores the energy flux (E_U + p_U) v_U of cell c at U_TMP[c*4 + 3]: the
// state's indexing applied to the 28-double scratch records, i.e. component 3
// of scratch slot c mod 7 of cell c/7.  With the serial row-major loop the
// target cell is already solved; for c mod 7 == 2 the store replaces the
// energy component of that cell's Y-face flux (slot 2), which the Y update
// then uses.  The sweep reproduces this in pull form: the Y face of cell c'
// recomputes the solve of its only possible source, cell 7 c' + 2.
//
// That solve reads the face states the reference's scratch slots hold at
// that point (MUSCL_Scheme.cpp / MHM_Scheme.cpp / Godunov_Scheme.cpp loop
// ranges, with the harness's zero-initialised scratch): slot 5 (U_D) is the
// Y reconstruction for rows [ng-1, N-1), else the X stage's U_L (columns
// [il0, M-1), il0 = ng-1 for MHM and 1 otherwise; MHM-predicted), else 0;
// slot 6 (U_U) the Y reconstruction for rows [0, N-2), else the X stage's
// U_R (columns [0, M-2)), else 0; MHM then predicts each slot in its row
// range from the fluxes of both.  Returns whether the branch fires at (i, j)
// and the value it stores.
template <int SCH, int LIM>
__device__ bool pvrs_stray_source(const double *__restrict__ U, long long P, int pitch, int M, int N, int ng,
                                  double g, double dt, double dx, double dy, int i, int j, double *value)
{
    auto cell = [&](int ii, int jj, double v[4]) {
#pragma unroll
        for (int k = 0; k < 4; k++)
            v[k] = U[k * P + (long long)jj * pitch + ii];
    };
    const int il0 = (SCH == MHM) ? ng - 1 : 1;
    const bool x5 = i >= il0 && i < M - 1, x6 = i < M - 2;
    const bool y5 = j >= ng - 1 && j < N - 1, y6 = j < N - 2;
    double s5[4] = {0.0, 0.0, 0.0, 0.0}, s6[4] = {0.0, 0.0, 0.0, 0.0};
    if (!y5 || !y6)
    {
        // the X stage's U_L and U_R at (i, j): MUSCL_Scheme.cpp:30-60 / MHM_Scheme.cpp:28-96
        double a[4], b[4], c[4], d[4];
        if (x5 || x6)
            cell(i, j, b);
        if (x5)
        {
            cell(i - 1, j, a);
            cell(i + 1, j, c);
#pragma unroll
            for (int k = 0; k < 4; k++)
                s5[k] = (SCH == GODUNOV) ? b[k] : b[k] + half_slope<LIM>(b[k], a[k], c[k], b[k]);
        }
        if (x6)
        {
            cell(i + 1, j, c);
            cell(i + 2, j, d);
#pragma unroll
            for (int k = 0; k < 4; k++)
                s6[k] = (SCH == GODUNOV) ? c[k] : c[k] - half_slope<LIM>(d[k], c[k], c[k], b[k]);
        }
        if (SCH == MHM)
        {
            double FL[4], FR[4];
            flux_x(s5, g, FL);
            flux_x(s6, g, FR);
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                double dd = 0.5 * (FL[k] - FR[k]) * dt / dx;
                if (x5)
                    s5[k] = s5[k] + dd;
                if (x6)
                    s6[k] = s6[k] + dd;
            }
        }
    }
    if (y5 || y6)
    {
        // the Y stage: MUSCL_Scheme.cpp:91-121 / MHM_Scheme.cpp:98-183
        double a[4], b[4], c[4], d[4];
        cell(i, j, b);
        cell(i, j + 1, c);
        if (y5)
        {
            cell(i, j - 1, a);
#pragma unroll
            for (int k = 0; k < 4; k++)
                s5[k] = (SCH == GODUNOV) ? b[k] : b[k] + half_slope<LIM>(b[k], a[k], c[k], b[k]);
        }
        if (y6)
        {
            cell(i, j + 2, d);
#pragma unroll
            for (int k = 0; k < 4; k++)
                s6[k] = (SCH == GODUNOV) ? c[k] : c[k] - half_slope<LIM>(d[k], c[k], c[k], b[k]);
        }
    }
    if (SCH == MHM)
    {
        double FL[4], FR[4];
        flux_y(s5, g, FL);
        flux_y(s6, g, FR);
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            double dd = 0.5 * (FL[k] - FR[k]) * dt / dy;
            if (y5)
                s5[k] = s5[k] + dd;
            if (y6)
                s6[k] = s6[k] + dd;
        }
    }
    double G[4], stray = 0.0;
    if (!(pvrs_y(s5, s6, g, G, &stray) & 8))
        return false;
    *value = stray;
    return true;
}

// One X face: states from four cells, MHM predictor, Riemann solver.
template <int SCH, int RIE, int LIM>
__device__ __forceinline__ void x_face(const double c0[4], const double c1[4], const double c2[4], const double c3[4],
                                       const GridDesc &g, double dt, double F[4])
{
    double UL[4], UR[4];
    face_states<SCH, LIM>(c0, c1, c2, c3, UL, UR);
    if (SCH == MHM)
        mhm_predict<1>(UL, UR, g, dt);
    if (RIE == PVRS)
        pvrs_x(UL, UR, g.gamma, F);
    else if (RIE == SW)
        strict_sw<1>(UL, UR, g, F);
    else
        strict_hll<1>(UL, UR, g, F);
}

// One Y face.  Returns the mask of components that keep the X-face flux of
// the same cell (all four for HLL with S_D >= 0, component 3 for the PVRS
// branch at :547-550, none otherwise).
template <int SCH, int RIE, int LIM>
__device__ __forceinline__ int y_face(const double c0[4], const double c1[4], const double c2[4], const double c3[4],
                                      const GridDesc &g, double dt, double G[4], double *stray)
{
    double UD[4], UU[4];
    face_states<SCH, LIM>(c0, c1, c2, c3, UD, UU);
    if (SCH == MHM)
        mhm_predict<2>(UD, UU, g, dt);
    if (RIE == PVRS)
        return pvrs_y(UD, UU, g.gamma, G, stray);
    if (RIE == SW)
    {
        strict_sw<2>(UD, UU, g, G);
        return 0;
    }
    return strict_hll<2>(UD, UU, g, G) ? 0 : 0xF;
}

} // namespace ibtfo
