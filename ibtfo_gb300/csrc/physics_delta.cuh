// Face fluxes of the FP32 form in difference form, for the HLL_Toro key.
//
// The plain FP32 face solve rounds each flux to about 1e-7 of its size, and
// the update takes the difference of two such fluxes, which in smooth flow is
// a hundred to a thousand times smaller than either: each step then adds an
// error of about 1e-7 of the flux to every cell that is not in uniform flow.
// Over thousands of steps in the unsteady wake of a body this is the error
// that separates an FP32 run from its FP64 twin.  Here no full-size flux is
// ever formed.  A face between cells a (left / lower) and b stores
//   P = F_face - F(U_a)   and   Q = F_face - F(U_b),
// and cell i updates with  F_east - F_west = P_east - Q_west  (the same
// value in exact arithmetic).  Every quantity is built from differences of
// the compensated (hi, lo) state, which are accurate to FP32 rounding of the
// difference itself:
//   F(U_b) - F(U_a) and F(U_face) - F(U_cell)  by delta_flux (the product
//   rule on the primitive variables, below), and
//   HLL:  F_face - F(U_a) = w_L dF_L + w_R (dF + dF_R) + (S_L S_R / (S_R - S_L)) (U_R - U_L)
//   with w_L = S_R / (S_R - S_L), w_R = -S_L / (S_R - S_L), so that rounding
//   errors are relative to these small terms, not to F.  The wave speeds
//   (Toro's PVRS estimates, as hll_plain) multiply small quantities only and
//   are formed from the FP32 face states.
// Two faces are solved at once in packed FP32 arithmetic (one instruction for
// two operations, each half rounding as the single one does): a third fewer
// instructions (vortex 2048^2, first stage: 158.7 M -> 110.5 M warp instructions).
// The bits are those of the single form.  The gain in time is smaller, since
// the registers of two faces leave 15 warps per SM, not 24 (issue slots used 69%
// -> 51%).  With the staging
// of sweep_tile32_delta, per step: cylinder 1800x1100 MUSCL + RK2 214-216 ->
// 192-197 us, vortex MHM + RK2 2048^2 460 -> 449 us, 4096^2 1.70 -> 1.65 ms.
// The algorithm is HLL_Toro's (MUSCL / MHM / Godunov reconstruction with the
// limiter, the positivity fallback and the same HLL flux); only the order of
// evaluation differs.
#pragma once

#include "physics_fast.cuh"

namespace ibtfo {

// two floats in one 64-bit register pair
struct F2
{
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float x, float y)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ float lo(F2 a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float hi(F2 a) { return __uint_as_float((unsigned)(a.v >> 32)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b)
{
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a) { return F2{a.v ^ 0x8000000080000000ull}; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// a where the half's condition holds, else b
__device__ __forceinline__ F2 choose(bool c0, bool c1, F2 a, F2 b)
{
    return f2(c0 ? lo(a) : lo(b), c1 ? hi(a) : hi(b));
}
__device__ __forceinline__ F2 rcp2(F2 x) // rcp_t of each half
{
    const F2 y = f2(rcp_estimate(lo(x)), rcp_estimate(hi(x)));
    return fma2(y, fma2(-x, y, f2(1.0f)), y);
}
__device__ __forceinline__ F2 sqrt2(F2 x) { return f2(sqrt_t(lo(x)), sqrt_t(hi(x))); }
__device__ __forceinline__ F2 minmod2(F2 a, F2 b)
{
    const F2 p = a * b;
    const float a0 = lo(a), a1 = hi(a), b0 = lo(b), b1 = hi(b);
    return f2((lo(p) > 0.0f) ? ((fabsf(a0) > fabsf(b0)) ? b0 : a0) : 0.0f,
              (hi(p) > 0.0f) ? ((fabsf(a1) > fabsf(b1)) ? b1 : a1) : 0.0f);
}

// gas constants in both halves
struct GasConst2
{
    F2 g, gm1, c1, c2;
    float igm1;
    __device__ __forceinline__ explicit GasConst2(const GridDesc &d)
        : g(f2(d.gf)), gm1(f2(d.gm1f)), c1(f2(d.c1f)), c2(f2(d.c2f)), igm1(d.igm1f)
    {
    }
};

// reciprocal density, velocities and pressure of a base state
struct DeltaBase
{
    F2 ir, un, ut, p;
};

template <int NRM>
__device__ __forceinline__ DeltaBase delta_base(const F2 U[4], const GasConst2 &K)
{
    DeltaBase b;
    b.ir = rcp2(U[0]);
    b.un = U[NRM] * b.ir;
    b.ut = U[3 - NRM] * b.ir;
    b.p = K.gm1 * fma2(f2(-0.5f), fma2(U[NRM], b.un, U[3 - NRM] * b.ut), U[3]);
    return b;
}

// whether a state has positive density and an internal energy p / (gamma - 1)
// above 1e-6 of E (NaN fails)
__device__ __forceinline__ bool physical_pressure(float r, float p, float E, const GasConst2 &K)
{
    return r > 0.0f && p * K.igm1 > 1e-6f * fabsf(E);
}

// dF = F(U_a + d) - F(U_a), normal direction NRM, from the base state U_a
// (FP32 values, velocities and pressure in `a`), the difference d and
// irb = 1 / (rho_a + d rho):
//   du_n = (d m_n - u_n d rho) / rho_b          (u = m / rho)
//   d(m_n u_n) = m_nb du_n + u_na d m_n,  d(m_t u_t) = m_tb du_t + u_ta d m_t
//   dp = (gamma - 1) (dE - (d(m_n u_n) + d(m_t u_t)) / 2)
//   dF = (d m_n, d(m_n u_n) + dp, m_tb du_n + u_na d m_t, (E_b + p_b) du_n + u_na (dE + dp))
// (components in state order; exact identities, so the rounding is relative
// to the differences).
template <int NRM>
__device__ __forceinline__ void delta_flux(const F2 Ua[4], const DeltaBase &a, const F2 d[4], F2 irb,
                                           const GasConst2 &K, F2 dF[4])
{
    const F2 dun = fma2(-a.un, d[0], d[NRM]) * irb;
    const F2 dut = fma2(-a.ut, d[0], d[3 - NRM]) * irb;
    const F2 mnb = Ua[NRM] + d[NRM], mtb = Ua[3 - NRM] + d[3 - NRM];
    const F2 dnn = fma2(mnb, dun, a.un * d[NRM]);
    const F2 dtt = fma2(mtb, dut, a.ut * d[3 - NRM]);
    const F2 e = fma2(f2(-0.5f), dnn + dtt, d[3]); // dp / (gamma - 1)
    dF[0] = d[NRM];
    dF[NRM] = fma2(K.gm1, e, dnn);
    dF[3 - NRM] = fma2(mtb, dun, a.un * d[3 - NRM]);
    dF[3] = fma2((Ua[3] + d[3]) + fma2(K.gm1, e, a.p), dun, a.un * fma2(K.gm1, e, d[3]));
}

// two faces in difference form: cells c0 c1 | c2 c3 across each (hi and lo
// parts), normal NRM; P = F_face - F(c1), Q = F_face - F(c2).  hp = dt/(2h)
// for the MHM predictor.  The reciprocal densities of the cell and face
// states serve both the primitive variables and the flux differences, and
// the positivity tests read the primitive variables.
// ld(n, k): plane k (0-3 hi, 4-7 lo) of cell n, both faces.
template <int SCH, int LIM, int NRM, typename Load>
__device__ __forceinline__ void face_delta(const Load &ld, const GasConst2 &K, float hp, F2 P[4], F2 Q[4])
{
    F2 D1[4], dL[4], dR[4], UcL[4], UcR[4], UL[4], UR[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
        // differences of the compensated states: hi parts first (exact for
        // neighbouring values), then the lo parts
        const F2 h0 = ld(0, k), h1 = ld(1, k), h2 = ld(2, k), h3 = ld(3, k);
        const F2 l0 = ld(0, 4 + k), l1 = ld(1, 4 + k), l2 = ld(2, 4 + k), l3 = ld(3, 4 + k);
        const F2 D0 = (h1 - h0) + (l1 - l0);
        D1[k] = (h2 - h1) + (l2 - l1);
        const F2 D2 = (h3 - h2) + (l3 - l2);
        UcL[k] = h1 + l1;
        UcR[k] = h2 + l2;
        if (SCH == GODUNOV)
            dL[k] = dR[k] = f2(0.0f);
        else if (LIM == VANLEER)
        {
            dL[k] = f2(0.5f) * f2(vanleer_t<float>(lo(D0), lo(UcR[k]), lo(UcL[k])),
                                  vanleer_t<float>(hi(D0), hi(UcR[k]), hi(UcL[k])));
            dR[k] = f2(-0.5f) * f2(vanleer_t<float>(lo(D2), lo(UcR[k]), lo(UcL[k])),
                                   vanleer_t<float>(hi(D2), hi(UcR[k]), hi(UcL[k])));
        }
        else
        {
            dL[k] = f2(0.5f) * minmod2(D0, D1[k]);
            dR[k] = f2(-0.5f) * minmod2(D2, D1[k]);
        }
        UL[k] = h1 + (l1 + dL[k]);
        UR[k] = h2 + (l2 + dR[k]);
    }
    const DeltaBase bL = delta_base<NRM>(UcL, K), bR = delta_base<NRM>(UcR, K);
    F2 dF[4], fL[4], fR[4];
    delta_flux<NRM>(UcL, bL, D1, bR.ir, K, dF);
    DeltaBase L = bL, R = bR;
    F2 rL = UcL[0], rR = UcR[0];
    if (SCH == GODUNOV)
    {
#pragma unroll
        for (int k = 0; k < 4; k++)
            fL[k] = fR[k] = f2(0.0f);
    }
    else
    {
        if (SCH == MHM)
        {
            // U_L, U_R += (dt / 2h) (F(U_L) - F(U_R)), F(U_L) - F(U_R) = dF_L - dF - dF_R
            delta_flux<NRM>(UcL, bL, dL, rcp2(UL[0]), K, fL);
            delta_flux<NRM>(UcR, bR, dR, rcp2(UR[0]), K, fR);
            const F2 hp2 = f2(hp);
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                const F2 x = (fL[k] - dF[k]) - fR[k];
                dL[k] = fma2(hp2, x, dL[k]);
                dR[k] = fma2(hp2, x, dR[k]);
                UL[k] = ld(1, k) + (ld(1, 4 + k) + dL[k]);
                UR[k] = ld(2, k) + (ld(2, 4 + k) + dR[k]);
            }
        }
        L = delta_base<NRM>(UL, K);
        R = delta_base<NRM>(UR, K);
        const bool ok0 = physical_pressure(lo(UL[0]), lo(L.p), lo(UL[3]), K) &&
                         physical_pressure(lo(UR[0]), lo(R.p), lo(UR[3]), K);
        const bool ok1 = physical_pressure(hi(UL[0]), hi(L.p), hi(UL[3]), K) &&
                         physical_pressure(hi(UR[0]), hi(R.p), hi(UR[3]), K);
        if (!(ok0 && ok1))
        {
            // positivity fallback of a face between two physical cells: the
            // first-order pair (the two cell averages; dL = dR = 0 makes the
            // flux differences below zero)
            const bool keep0 = ok0 || !(physical_pressure(lo(UcL[0]), lo(bL.p), lo(UcL[3]), K) &&
                                        physical_pressure(lo(UcR[0]), lo(bR.p), lo(UcR[3]), K));
            const bool keep1 = ok1 || !(physical_pressure(hi(UcL[0]), hi(bL.p), hi(UcL[3]), K) &&
                                        physical_pressure(hi(UcR[0]), hi(bR.p), hi(UcR[3]), K));
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                dL[k] = choose(keep0, keep1, dL[k], f2(0.0f));
                dR[k] = choose(keep0, keep1, dR[k], f2(0.0f));
            }
            UL[0] = choose(keep0, keep1, UL[0], UcL[0]);
            UR[0] = choose(keep0, keep1, UR[0], UcR[0]);
            L.ir = choose(keep0, keep1, L.ir, bL.ir), R.ir = choose(keep0, keep1, R.ir, bR.ir);
            L.un = choose(keep0, keep1, L.un, bL.un), R.un = choose(keep0, keep1, R.un, bR.un);
            L.p = choose(keep0, keep1, L.p, bL.p), R.p = choose(keep0, keep1, R.p, bR.p);
        }
        rL = UL[0];
        rR = UR[0];
        delta_flux<NRM>(UcL, bL, dL, L.ir, K, fL);
        delta_flux<NRM>(UcR, bR, dR, R.ir, K, fR);
    }
    // Toro's PVRS wave-speed estimates from the face states (hll_plain)
    const F2 gL = K.g * L.ir, gR = K.g * R.ir;
    const F2 aL = sqrt2(gL * L.p), aR = sqrt2(gR * R.p);
    F2 ps = fma2(f2(0.5f), L.p + R.p, f2(0.125f) * (L.un - R.un) * ((rL + rR) * (aL + aR)));
    ps = f2(fmaxf(lo(ps), 0.0f), fmaxf(hi(ps), 0.0f)); // NaN: 0
    const F2 t = K.c1 * ps;
    const F2 qL = sqrt2(gL * fma2(K.c2, L.p, t)), qR = sqrt2(gR * fma2(K.c2, R.p, t));
    const F2 S_L = L.un - choose(lo(ps) > lo(L.p), hi(ps) > hi(L.p), qL, aL);
    const F2 S_R = R.un + choose(lo(ps) > lo(R.p), hi(ps) > hi(R.p), qR, aR);
    const F2 inv = rcp2(S_R - S_L);
    const F2 wr = -S_L * inv, wl = S_R * inv, c = S_L * S_R * inv;
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
        const F2 dU = (D1[k] + dR[k]) - dL[k]; // U_R - U_L
        P[k] = fma2(wl, fL[k], fma2(wr, dF[k] + fR[k], c * dU));
        Q[k] = P[k] - dF[k];
    }
    const bool l0 = lo(S_L) >= 0.0f, l1 = hi(S_L) >= 0.0f, r0 = lo(S_R) <= 0.0f, r1 = hi(S_R) <= 0.0f;
    if (l0 || l1 || r0 || r1)
    {
        // supersonic: F_face = F(U_L) = F(c1) + dF_L, or F(U_R) = F(c2) + dF_R
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            P[k] = choose(r0, r1, dF[k] + fR[k], P[k]);
            Q[k] = choose(r0, r1, fR[k], Q[k]);
            P[k] = choose(l0, l1, fL[k], P[k]);
            Q[k] = choose(l0, l1, fL[k] - dF[k], Q[k]);
        }
    }
}

} // namespace ibtfo
