// The fp64_fast faces: the algorithms of physics_fast.cuh in the fewest FP64
// instructions.
//
// What bounds the FP64 sweeps is the FP64 unit, one per SM, which takes 16
// clocks for a warp instruction: an FP64 instruction costs as much as 64
// integer or FP32 ones, and a partly filled warp as much as a full one.
// Three things follow:
//   * reciprocals and square roots are taken on the integer and FP32 pipes
//     (int64math.cuh), which the faces leave idle;
//   * comparisons and the positivity tests read bit patterns;
//   * the HLL flux is taken as a correction to one side's flux
//     (hll_combine64: 22 instructions, 27 before), and
//     Steger-Warming's sums over the three waves are regrouped around
//     T = 2 (gamma - 1) l1 + l3 + l4 (43 per state instead of 77).
// Channel 2048x1024, MUSCL + HLL, one sweep: 161.4 M -> 92.7 M FP64 thread
// instructions, 372 -> 223 us, the unit busy for 83% of the active cycles.
// Also tried: the products too on the integer pipes, exactly (four 32-bit
// multiplies and the rounding, about 40 instructions each): the same bits, but
// the code outgrows the instruction cache (fp64_fast 7.8 -> 8.6 ms for 32
// steps, strict 5.5 -> 6.5 for 12).
#pragma once

#include "physics_fast.cuh"

namespace ibtfo {

// a state with its primitive variables across a face of normal NRM
struct Prim64
{
    double r, ir, mn, mt, E, un, ei, p; // ei = E - rho (u^2 + v^2) / 2, p = (gamma - 1) ei
};

template <int NRM>
__device__ __forceinline__ Prim64 prim64(const double U[4], const GasConst<double> &K)
{
    Prim64 s;
    s.r = U[0];
    s.mn = U[NRM];
    s.mt = U[3 - NRM];
    s.E = U[3];
    s.ir = rcp_t(s.r);
    s.un = s.mn * s.ir;
    s.ei = fma(-0.5, fma(s.mn, s.un, s.mt * (s.mt * s.ir)), s.E);
    s.p = K.gm1 * s.ei;
    return s;
}

// flux of one state normal to the face; m_t u_n is the tangential momentum flux
template <int NRM>
__device__ __forceinline__ void flux64(const Prim64 &s, double F[4])
{
    F[0] = s.mn;
    F[NRM] = fma(s.mn, s.un, s.p);
    F[3 - NRM] = s.mt * s.un;
    F[3] = (s.E + s.p) * s.un;
}

// The HLL combination of two states with wave speeds S_L < 0 < S_R, taken from
// one state A towards the other, B: with S the wave speed on B's side and w the
// magnitude of the one on A's side over S_R - S_L,
//   F = F_A + w ((F_B - F_A) - S (U_B - U_A)).
// A is the state of the larger weight, 1 - w >= 1/2 (a comparison of
// magnitudes, and selections, on the integer pipe).  The correction is small in
// smooth flow, so that a component rounds little beyond F_A itself: half the
// r.m.s. error of the weighted form w_L F_L + w_R F_R + w_U (U_R - U_L) there,
// no more at strong jumps (tests/test_fast64_faces_cpu.py), in 22 instructions
// where that form takes 25 to 27.  A shorter one in 17, A U_L + B U_R + ... from
// F_K - S_K U_K = +-c_K U_K + p_K (0, 1, 0, u_K), rounds against c U and not against
// the flux (mass flux at a Mach number up to 0.03: 38 times the error).
template <int NRM>
__device__ __forceinline__ void hll_combine64(const Prim64 &L, const Prim64 &R, double S_L, double S_R, double F[4])
{
    if (ge0(S_L))
        flux64<NRM>(L, F);
    else if (le0(S_R))
        flux64<NRM>(R, F);
    else
    {
        const double inv = rcp_t(S_R - S_L);
        const bool left = magnitude_bits(S_L) < magnitude_bits(S_R);
        const Prim64 A = left ? L : R, B = left ? R : L;
        // (a selected negation would be an FP64 addition)
        const double S = left ? S_R : S_L, w = magnitude(left ? S_L : S_R) * inv;
        const double dm = B.mn - A.mn; // also the difference of the mass fluxes
        const double FN = fma(A.mn, A.un, A.p), FT = A.mt * A.un, FE = (A.E + A.p) * A.un;
        F[0] = fma(w, fma(-S, B.r - A.r, dm), A.mn);
        F[NRM] = fma(w, fma(-S, dm, fma(B.mn, B.un, B.p) - FN), FN);
        F[3 - NRM] = fma(w, fma(-S, B.mt - A.mt, fma(B.mt, B.un, -FT)), FT);
        F[3] = fma(w, fma(-S, B.E - A.E, fma(B.E + B.p, B.un, -FE)), FE);
    }
}

// HLL face flux (HLL/Riemann_solver.cpp:131-169 X, :202-235 Y).  For Y,
// returns false when S_D >= 0 (the reference keeps the X-face flux).
// With q_K = gamma / (16 rho_K), a_K / 4 = sqrt(q_K p_K) and
// W = 2 p* = p_L + p_R + (u_L - u_R) (rho_L + rho_R) (a_L + a_R) / 4:
// c_K = sqrt((gamma / rho_K) (c1 p* + c2 p_K)) = sqrt(q_K (8 c1 W + 16 c2 p_K)).
template <int NRM>
__device__ __forceinline__ bool hll64(const double UL[4], const double UR[4], const GasConst<double> &K, double F[4])
{
    const Prim64 L = prim64<NRM>(UL, K), R = prim64<NRM>(UR, K);
    const double qL = K.g16 * L.ir, qR = K.g16 * R.ir;
    const double W = fma(L.un - R.un, (L.r + R.r) * (sqrt_t(qL * L.p) + sqrt_t(qR * R.p)), L.p + R.p);
    const double t = K.c1x8 * W;
    const double cL = sqrt_t(qL * fma(K.c2x16, L.p, t));
    const double S_L = L.un - cL;
    if (NRM == 2 && ge0(S_L))
        return false;
    const double cR = sqrt_t(qR * fma(K.c2x16, R.p, t));
    hll_combine64<NRM>(L, R, S_L, R.un + cR, F);
    return true;
}

// w > 2 p for a w that is zero, normal or +Inf (not NaN): doubles of one sign
// order like their bits, and halving a normal number takes one from its exponent
// (w >= 0, so that the difference cannot overflow).  True for every finite
// negative p and -0; false for p = +Inf and for NaNs without the sign bit (-Inf and
// the other NaNs: either; the sound speed is NaN then, and the wave speed with
// it).  w = +Inf counts as 2^1024: not above twice a p of 2^1023 or more.
__device__ __forceinline__ bool exceeds_twice(double w, double p)
{
    return __double_as_longlong(w) - 0x0010000000000000LL > __double_as_longlong(p);
}

// HLL with Toro's wave-speed estimates (hll_plain: p* >= 0, q_K = 1 for p* <= p_K)
template <int NRM>
__device__ __forceinline__ void hll_toro64(const Prim64 &L, const Prim64 &R, const GasConst<double> &K, double F[4])
{
    const double gL = K.g * L.ir, gR = K.g * R.ir;
    const double aL = sqrt_t(gL * L.p), aR = sqrt_t(gR * R.p);
    double W = fma(0.25 * (L.un - R.un), (L.r + R.r) * (aL + aR), L.p + R.p); // 2 p*
    const long long bw = __double_as_longlong(W);
    W = (bw > 0 && bw <= 0x7ff0000000000000LL) ? W : 0.0;
    const double t = K.c1h * W;
    double cL = aL, cR = aR;
    if (exceeds_twice(W, L.p))
        cL = sqrt_t(gL * fma(K.c2, L.p, t));
    if (exceeds_twice(W, R.p))
        cR = sqrt_t(gR * fma(K.c2, R.p, t));
    hll_combine64<NRM>(L, R, L.un - cL, R.un + cR, F);
}

// Contact-restoring HLLC with Toro's wave speeds (hllc_toro), from the primitive variables
template <int NRM>
__device__ __forceinline__ void hllc_toro64(const Prim64 &L, const Prim64 &R, const GasConst<double> &K, double F[4])
{
    const double gL = K.g * L.ir, gR = K.g * R.ir;
    const double aL = sqrt_t(gL * L.p), aR = sqrt_t(gR * R.p);
    double W = fma(0.25 * (L.un - R.un), (L.r + R.r) * (aL + aR), L.p + R.p);
    const long long bw = __double_as_longlong(W);
    W = (bw > 0 && bw <= 0x7ff0000000000000LL) ? W : 0.0;
    const double t = K.c1h * W;
    double cL = aL, cR = aR;
    if (exceeds_twice(W, L.p))
        cL = sqrt_t(gL * fma(K.c2, L.p, t));
    if (exceeds_twice(W, R.p))
        cR = sqrt_t(gR * fma(K.c2, R.p, t));
    const double S_L = L.un - cL, S_R = R.un + cR;
    if (ge0(S_L))
    {
        flux64<NRM>(L, F);
        return;
    }
    if (le0(S_R))
    {
        flux64<NRM>(R, F);
        return;
    }
    // rho_K (S_K - u_K): -rho_L c_L and rho_R c_R
    const double mL = L.r * (S_L - L.un), mR = R.r * (S_R - R.un);
    const double S_s = (R.p - L.p + L.un * mL - R.un * mR) * rcp_t(mL - mR);
    const bool left = ge0(S_s);
    const Prim64 s = left ? L : R;
    const double S = left ? S_L : S_R, m = left ? mL : mR;
    const double fac = m * rcp_t(S - S_s);
    double Fk[4];
    flux64<NRM>(s, Fk);
    F[0] = Fk[0] + S * (fac - s.r);
    F[NRM] = Fk[NRM] + S * (fac * S_s - s.mn);
    F[3 - NRM] = Fk[3 - NRM] + S * (fac * (s.mt * s.ir) - s.mt);
    F[3] = Fk[3] + S * (fac * (s.E * s.ir + (S_s - s.un) * (S_s + s.p * rcp_t(m))) - s.E);
}

// One side of the Steger-Warming splitting (StegerWarming/Riemann_solver.cpp:
// 173-234 X, :262-325 Y), added to F.  With L_k = lambda_k +- sqrt(lambda_k^2
// + delta^2) (twice the reference's), T = 2 (gamma - 1) L1 + L3 + L4,
// X = a (L4 - L3), w = rho / (4 gamma), k = rho |u|^2 and the internal energy
// ei = rho a^2 / (gamma (gamma - 1)):
//   F = (w T, u_n w T + w X, u_t w T, k/2 T/(4 gamma) + ei/4 (L3 + L4) + u_n w X)
// Each of T, a and ei is rounded as often as in the plain form or less: ei is
// taken from E and not from E / rho, and the two small wave speeds are added
// first in T (a sum around L3 + L4 had 9% more error in the mass flux of one
// side; tests/test_fast64_faces_cpu.py).
template <int NRM, int SIGN>
__device__ __forceinline__ void sw_split64(const double U[4], const GasConst<double> &K, double F[4])
{
    const double ir = rcp_t(U[0]);
    const double un = U[NRM] * ir, ut = U[3 - NRM] * ir;
    const double k = fma(U[NRM], un, U[3 - NRM] * ut);
    const double ei = fma(-0.5, k, U[3]);
    const double a = sqrt_t((K.g * ir) * (K.gm1 * ei));
    const double d2 = 1e-12; // delta = 1e-6 (:193)
    auto lam = [&](double x) {
        const double r = sqrt_t(fma(x, x, d2));
        return SIGN > 0 ? x + r : x - r;
    };
    const double l1 = lam(un), l3 = lam(un - a), l4 = lam(un + a);
    // SIGN > 0: l3 is the small one below Mach 1; SIGN < 0: l4
    const double T = SIGN > 0 ? fma(K.gm1x2, l1, l3) + l4 : fma(K.gm1x2, l1, l4) + l3, X = a * (l4 - l3);
    const double t = K.ig4 * T, wT = U[0] * t, wX = (K.ig4 * U[0]) * X;
    const double g2 = fma(0.5 * k, t, fma(un, wX, (0.25 * ei) * (l3 + l4)));
    F[0] = (SIGN > 0) ? wT : F[0] + wT;
    F[NRM] = (SIGN > 0) ? fma(un, wT, wX) : F[NRM] + fma(un, wT, wX);
    F[3 - NRM] = (SIGN > 0) ? ut * wT : fma(ut, wT, F[3 - NRM]);
    F[3] = (SIGN > 0) ? g2 : F[3] + g2;
}

// MHM predictor with h2 = dt / (2 h) (mhm_predict_fast)
template <int NRM>
__device__ __forceinline__ void mhm_predict64(double UL[4], double UR[4], const GasConst<double> &K, double h2)
{
    const Prim64 L = prim64<NRM>(UL, K), R = prim64<NRM>(UR, K);
    double FL[4], FR[4];
    flux64<NRM>(L, FL);
    flux64<NRM>(R, FR);
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
        const double d = FL[k] - FR[k];
        UL[k] = fma(h2, d, UL[k]);
        UR[k] = fma(h2, d, UR[k]);
    }
}

// x > f |E| for a threshold f < 2^-(DROP + 0.1), settled on the high words
// where x / |E| is well above it: a high word is a number's exponent and the
// leading bits of its significand, so that a difference above -(DROP << 20)
// means x / |E| > 2^-(DROP + 0.1); closer values are compared in FP64
static __device__ __noinline__ bool above_fraction_fp64(double x, double E, double f) { return x > f * fabs(E); }
template <int DROP>
__device__ __forceinline__ bool above_fraction(double x, double E, double f)
{
    const int hx = __double2hiint(x), hE = __double2hiint(E) & 0x7fffffff;
    if (hx >= 0x00100000 && hx < 0x7ff00000 && hE < 0x7ff00000 && hx - hE >= -(DROP << 20))
        return true;
    return above_fraction_fp64(x, E, f);
}
// positive density and an internal energy above 1e-6 E (physical())
__device__ __forceinline__ bool physical64(const Prim64 &s)
{
    const long long b = __double_as_longlong(s.r);
    return b > 0 && b <= 0x7ff0000000000000LL && above_fraction<18>(s.ei, s.E, 1e-6);
}

// velocity and internal energy of a cell's state
struct Cell64
{
    double ir, u, v, ei;
};
__device__ __forceinline__ Cell64 cell64(const double U[4])
{
    Cell64 c;
    c.ir = rcp_t(U[0]);
    c.u = U[1] * c.ir;
    c.v = U[2] * c.ir;
    c.ei = fma(-0.5, fma(U[1], c.u, U[2] * c.v), U[3]);
    return c;
}

// the pressure floor (pressure_floor_energy) of an updated cell: raises U[3]
// and c.ei where the internal energy is below 1e-5 E
static __device__ __noinline__ double floored_energy(double rho, double ei, double E)
{
    const double f = 1e-5 * fabs(E);
    return (rho > 0.0 && !(ei >= f)) ? f : ei;
}
__device__ __forceinline__ void pressure_floor64(double U[4], Cell64 &c)
{
    if (above_fraction<15>(c.ei, U[3], 1e-5))
        return;
    const double f = floored_energy(U[0], c.ei, U[3]);
    if (__double_as_longlong(f) == __double_as_longlong(c.ei))
        return;
    U[3] = (U[3] - c.ei) + f;
    // a cell left NaN (a momentum that is, or E = -Inf) stays out of the CFL maximum
    c.ei = magnitude_bits(U[3]) <= 0x7ff0000000000000LL ? f : U[3];
}

// The primitive variables of a face's pair; a pair that is not physical
// between two cells that are takes the two cell averages
// (positivity_fallback).  The cells are looked at only then.
template <int NRM, bool SAFE>
__device__ __forceinline__ void face_prims64(const double c1[4], const double c2[4], const double UL[4],
                                             const double UR[4], const GasConst<double> &K, Prim64 &L, Prim64 &R)
{
    L = prim64<NRM>(UL, K);
    R = prim64<NRM>(UR, K);
    if (SAFE && !(physical64(L) && physical64(R)))
    {
        const Prim64 a = prim64<NRM>(c1, K), b = prim64<NRM>(c2, K);
        if (physical64(a) && physical64(b))
        {
            L = a;
            R = b;
        }
    }
}

// The flux from the pair (UL, UR) of a face between cells c1 and c2; false:
// the Y face keeps its slot's X-face flux (HLL only).  SAFE: the positivity
// fallback applies (the Toro keys, and every cut-cell solver).
template <int NRM, int RIE, bool SAFE>
__device__ __forceinline__ bool solve64(const double c1[4], const double c2[4], double UL[4], double UR[4],
                                        const GasConst<double> &K, double F[4])
{
    if constexpr (RIE == SW)
    {
        if (SAFE)
        {
            Prim64 L = prim64<NRM>(UL, K), R = prim64<NRM>(UR, K);
            if (!(physical64(L) && physical64(R)))
            {
                L = prim64<NRM>(c1, K), R = prim64<NRM>(c2, K);
                if (physical64(L) && physical64(R))
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        UL[k] = c1[k], UR[k] = c2[k];
            }
        }
        sw_split64<NRM, 1>(UL, K, F);
        sw_split64<NRM, -1>(UR, K, F);
        return true;
    }
    else if constexpr (RIE == HLLT || RIE == HLLCT)
    {
        Prim64 L, R;
        face_prims64<NRM, SAFE>(c1, c2, UL, UR, K, L, R);
        if constexpr (RIE == HLLT)
            hll_toro64<NRM>(L, R, K, F);
        else
            hllc_toro64<NRM>(L, R, K, F);
        return true;
    }
    else
        return hll64<NRM>(UL, UR, K, F);
}

// One face of the FP64 sweeps, normal NRM; returns the components of a Y face
// that keep the X-face flux of its slot (HLL: all, PVRS: the energy, whose
// stray value *stray receives)
template <int SCH, int RIE, int LIM, int NRM>
__device__ __forceinline__ int face64(const double c0[4], const double c1[4], const double c2[4], const double c3[4],
                                      const GasConst<double> &K, double h2, double F[4], double *stray)
{
    double UL[4], UR[4];
    face_states_fast<double, SCH, LIM>(c0, c1, c2, c3, UL, UR);
    if (SCH == MHM)
        mhm_predict64<NRM>(UL, UR, K, h2);
    if constexpr (RIE == PVRS)
    {
        if (NRM == 2)
            return pvrs_y(UL, UR, K.g, F, stray);
        pvrs_x(UL, UR, K.g, F);
        return 0;
    }
    else
        return solve64<NRM, RIE, safeguarded(RIE) && SCH != GODUNOV>(c1, c2, UL, UR, K, F) ? 0 : 0xF;
}

// One face of the FP64 cut-cell sweeps (ccm_face)
template <int NRM, int SCH, int RIE, int LIM>
__device__ __forceinline__ void ccm_face64(const double c0[4], const double c1[4], const double c2[4],
                                           const double c3[4], const GasConst<double> &K, double h2, bool first_order,
                                           double F[4])
{
    double UL[4], UR[4];
    if (first_order || SCH == GODUNOV)
    {
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            UL[k] = c1[k];
            UR[k] = c2[k];
        }
    }
    else
    {
        face_states_fast<double, SCH, LIM>(c0, c1, c2, c3, UL, UR);
        if (SCH == MHM)
            mhm_predict64<NRM>(UL, UR, K, h2);
    }
    // first-order pairs are the cell averages: the fallback changes nothing there
    solve64<NRM, RIE, SCH != GODUNOV>(c1, c2, UL, UR, K, F);
}

// The wall flux of the FP64 cut-cell sweeps (ccm_wall_flux)
template <int RIE>
__device__ __forceinline__ void ccm_wall_flux64(const double U[4], double nx, double ny, const GasConst<double> &K,
                                                double W[4])
{
    const double mn = U[1] * nx + U[2] * ny, mt = -U[1] * ny + U[2] * nx;
    double UL[4] = {U[0], mn, mt, U[3]}, UR[4] = {U[0], -mn, mt, U[3]}, F[4];
    solve64<1, RIE, false>(UL, UR, UL, UR, K, F);
    W[0] = 0.0;
    W[1] = F[1] * nx;
    W[2] = F[1] * ny;
    W[3] = 0.0;
}

// A cut cell's wall: its length and outward unit normal, from the aperture
// differences times the cell sides (nLx, nLy)
struct CutWall
{
    double L, nx, ny;
};
__device__ __forceinline__ CutWall cut_wall(double nLx, double nLy)
{
    CutWall w{sqrt_rn(nLx * nLx + nLy * nLy), 0.0, 0.0};
    if (w.L > 0.0)
    {
        const Divisor by_L = divisor(w.L);
        w.nx = divide_rn(nLx, by_L);
        w.ny = divide_rn(nLy, by_L);
    }
    return w;
}

// one component of a cut cell: (alpha U - dt/dx fx - dt/dy gy - dt/(dx dy) L W) / alpha,
// the quotients IEEE's (a product with a rounded reciprocal adds up to an ulp)
__device__ __forceinline__ double cut_update(const Divisor &by_alpha, double U, double lx, double fx, double ly,
                                             double gy, double lw, double W)
{
    return divide_rn(by_alpha.b * U - lx * fx - ly * gy - lw * W, by_alpha);
}

} // namespace ibtfo
