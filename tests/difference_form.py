"""One step of HLL_Toro in difference form (csrc/physics_delta.cuh), one face at a
time on whole arrays: in float32 the FP32 sweep's arithmetic up to fused
operations and the hardware's reciprocal and root, in float64 the same algorithm.
MUSCL or MHM with either limiter, walls (Regular), no immersed body; states whose
faces need no positivity fallback (checked)."""
import numpy as np


def _limited(a, P, Q, D1, limiter):
    T = D1.dtype.type
    if limiter == "VanLeer":  # the reference's macro: slope from the cells' values
        r = (a + T(1e-7)) / ((P - Q) + T(1e-7))
        return np.where(r > 0, (r * r + r) * P - Q / (r * r + T(1)), T(0))
    return np.where(a * D1 > 0, np.where(np.abs(a) > np.abs(D1), D1, a), T(0))


class _Base:
    def __init__(self, U, n, gm1):
        self.ir = U.dtype.type(1) / U[0]
        self.un, self.ut = U[n] * self.ir, U[3 - n] * self.ir
        self.p = gm1 * (U[3] - U.dtype.type(0.5) * (U[n] * self.un + U[3 - n] * self.ut))


def _flux_difference(Ua, a, d, irb, n, gm1):
    dun, dut = (d[n] - a.un * d[0]) * irb, (d[3 - n] - a.ut * d[0]) * irb
    mnb, mtb = Ua[n] + d[n], Ua[3 - n] + d[3 - n]
    dnn, dtt = mnb * dun + a.un * d[n], mtb * dut + a.ut * d[3 - n]
    dp = gm1 * (d[3] - Ua.dtype.type(0.5) * (dnn + dtt))
    F = np.empty_like(Ua)
    F[0], F[n], F[3 - n] = d[n], dnn + dp, mtb * dun + a.un * d[3 - n]
    F[3] = ((Ua[3] + d[3]) + (a.p + dp)) * dun + a.un * (d[3] + dp)
    return F


def _faces(h, l, n, scheme, limiter, gamma, hp):
    """(P, Q) of the faces between cells k + 1 and k + 2 along the last axis."""
    T = h.dtype.type
    m = h.shape[-1] - 3
    (h0, h1, h2, h3), (l0, l1, l2, l3) = ([x[..., k:k + m] for k in range(4)] for x in (h, l))
    g, gm1, half = T(gamma), T(gamma - 1), T(0.5)
    D0, D1, D2 = (h1 - h0) + (l1 - l0), (h2 - h1) + (l2 - l1), (h3 - h2) + (l3 - l2)
    UcL, UcR = h1 + l1, h2 + l2
    dL, dR = half * _limited(D0, UcR, UcL, D1, limiter), -half * _limited(D2, UcR, UcL, D1, limiter)
    UL, UR = h1 + (l1 + dL), h2 + (l2 + dR)
    bL, bR = _Base(UcL, n, gm1), _Base(UcR, n, gm1)
    dF = _flux_difference(UcL, bL, D1, bR.ir, n, gm1)
    if scheme == "MHM":
        x = (_flux_difference(UcL, bL, dL, T(1) / UL[0], n, gm1) - dF) - \
            _flux_difference(UcR, bR, dR, T(1) / UR[0], n, gm1)
        dL, dR = dL + hp * x, dR + hp * x
        UL, UR = h1 + (l1 + dL), h2 + (l2 + dR)
    L, R = _Base(UL, n, gm1), _Base(UR, n, gm1)
    assert min(UL[0].min(), UR[0].min()) > 0 and min((L.p / np.abs(UL[3])).min(), (R.p / np.abs(UR[3])).min()) > 1e-4
    fL, fR = _flux_difference(UcL, bL, dL, L.ir, n, gm1), _flux_difference(UcR, bR, dR, R.ir, n, gm1)
    c1, c2 = T((gamma + 1) / (2 * gamma)), T((gamma - 1) / (2 * gamma))
    gL, gR = g * L.ir, g * R.ir
    aL, aR = np.sqrt(gL * L.p), np.sqrt(gR * R.p)
    ps = np.maximum(half * (L.p + R.p) + T(0.125) * (L.un - R.un) * ((UL[0] + UR[0]) * (aL + aR)), T(0))
    SL = L.un - np.where(ps > L.p, np.sqrt(gL * (c2 * L.p + c1 * ps)), aL)
    SR = R.un + np.where(ps > R.p, np.sqrt(gR * (c2 * R.p + c1 * ps)), aR)
    inv = T(1) / (SR - SL)
    P = SR * inv * fL + (-SL * inv * (dF + fR) + SL * SR * inv * ((D1 + dR) - dL))
    Q = P - dF
    P, Q = np.where(SR <= 0, dF + fR, P), np.where(SR <= 0, fR, Q)
    return np.where(SL >= 0, fL, P), np.where(SL >= 0, fL - dF, Q)


def step(u, dx, dy, dt, scheme, limiter, dtype=np.float32, gamma=1.4):
    """The interior (n_y, n_x, 4) after one step from the state u (N, M, 4) with its two ghost layers filled."""
    T = np.dtype(dtype).type
    U = np.moveaxis(u, -1, 0)
    h = U.astype(dtype)
    l = (U - h.astype(np.float64)).astype(dtype)
    lx, ly = T(dt) * T(1 / dx), T(dt) * T(1 / dy)
    P, Q = _faces(h[:, 2:-2], l[:, 2:-2], 1, scheme, limiter, gamma, T(0.5) * lx)
    d = lx * (P[..., 1:] - Q[..., :-1])
    swap = lambda x: np.ascontiguousarray(x[:, :, 2:-2].transpose(0, 2, 1))  # noqa: E731
    P, Q = _faces(swap(h), swap(l), 2, scheme, limiter, gamma, T(0.5) * ly)
    d = d + (ly * (P[..., 1:] - Q[..., :-1])).transpose(0, 2, 1)
    new = (h[:, 2:-2, 2:-2].astype(np.float64) + l[:, 2:-2, 2:-2]) - d
    return np.moveaxis(new, 0, -1)
