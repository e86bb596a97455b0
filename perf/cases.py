"""Workloads of the solver for timing: what a user's program has it do, through
the package's public calls, with the same results in plain 64-bit torch.

A pass is a whole use of the solver: an initial state goes in from page-locked
host memory (or is built on the GPU from bodies and a shock), the loop steps,
and the state and the loop scalars come back.  Starting every pass from its
own initial state keeps the flow the same from pass to pass.  The host-array
pass instead keeps its state in the caller's array, as that call is meant to
be used, and the served pass sends requests through a running server.

Grids, solver keys and CFL numbers are those of ibtfo_gb300/cases.py, of the
tests and of bench.py, or odd sizes between them.
"""
import math
import random

import torch

import ibtfo_gb300 as ib
from ibtfo_gb300 import cases as plug

GAMMA = 1.4
FOREVER = 1e300


def listed():
    return [
        # the reference's own Sod tube in the default precision, to its end:
        # a grid of 160 tiles, where launches and their latency count
        dict(name="sod_tube", kind="tube", n_x=400, n_y=100, scheme="MUSCL", riemann="HLL", precision="fp64",
             time="SingleStep", cfl=0.5, t_end=0.2, steps=0),
        # the smallest grids: four states meeting at a point, odd sizes, a few
        # steps between outputs
        dict(name="quadrants_small", kind="quad", n_x=61, n_y=47, scheme="MHM", riemann="StegerWarming",
             precision="fp64_fast", time="SingleStep", cfl=0.4, steps=24),
        # the inclined channel at its benchmark size in the default precision
        # (the reference's expressions, ghost-fluid walls)
        dict(name="channel_fp64", kind="channel", n_x=2048, n_y=1024, scheme="MUSCL", riemann="HLLC",
             boundary="IDWBaseGFM", precision="fp64", time="SingleStep", cfl=0.45, steps=12),
        # the same in the precision the benchmark quotes
        dict(name="channel_fp64_fast", kind="channel", n_x=2048, n_y=1024, scheme="MUSCL", riemann="HLLC",
             boundary="IDWBaseGFM", precision="fp64_fast", time="SingleStep", cfl=0.45, steps=32),
        # a middle-sized channel with ragged tiles, the other wall method and
        # flux-vector splitting
        dict(name="channel_odd", kind="channel", n_x=777, n_y=389, scheme="MUSCL", riemann="StegerWarming",
             boundary="HBCGFM", precision="fp64_fast", time="SingleStep", cfl=0.45, steps=48),
        # the channel in the FP32 form (plain FP32 face solves)
        dict(name="channel_fp32", kind="channel", n_x=2048, n_y=1024, scheme="MUSCL", riemann="HLLC",
             boundary="IDWBaseGFM", precision="fp32c", time="SingleStep", cfl=0.45, steps=32),
        # a caller that keeps the state in its own page-locked array and has
        # it advanced step by step (bench.py's end-to-end number)
        dict(name="channel_host", kind="host", n_x=2048, n_y=1024, scheme="MUSCL", riemann="HLLC",
             boundary="IDWBaseGFM", precision="fp64_fast", time="SingleStep", cfl=0.45, steps=24),
        # smooth unsteady flow in FP64: the vortex pair's grid of bench.py
        dict(name="vortex_fp64_fast", kind="vortex", n_x=1024, n_y=1024, scheme="MHM", riemann="HLL_Toro",
             precision="fp64_fast", time="RK2", cfl=0.25, steps=8),
        # the vortex at its full size in the FP32 form: the largest state
        dict(name="vortex_fp32", kind="vortex", n_x=4096, n_y=4096, scheme="MHM", riemann="HLL_Toro",
             precision="fp32c", time="RK2", cfl=0.25, steps=24),
        # shock over a field of bodies, cut cells, FP32 form
        dict(name="obstacles_fp32", kind="obstacles", n_x=4096, n_y=2048, scheme="MUSCL", riemann="HLL_Toro",
             precision="fp32c", time="SingleStep", cfl=0.3, steps=24),
        # the same method in FP64 at a size a study would repeat many times
        dict(name="obstacles_fp64", kind="obstacles", n_x=1024, n_y=512, scheme="MUSCL", riemann="HLL_Toro",
             precision="fp64_fast", time="SingleStep", cfl=0.3, steps=24),
        # requests of uneven sizes through the server: set-up, batched steps,
        # read-back of each density
        dict(name="served_fp32", kind="served", requests=8, min_cells=128 * 128, max_cells=1024 * 1024,
             stream=42, scheme="MUSCL", riemann="HLL_Toro", precision="fp32c", time="RK2", cfl=0.45,
             crossings=0.1, n_x=0, n_y=0, steps=0),
    ]


def draw(rng):
    kind = rng.choice(["tube", "quad", "quad", "channel", "channel", "channel", "host", "vortex", "vortex",
                       "obstacles", "served"])

    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "served":
        lo = between(96, 200)
        return dict(kind=kind, requests=rng.randint(3, 8), min_cells=lo * lo, max_cells=between(256, 900) ** 2,
                    stream=rng.randrange(1 << 20), scheme="MUSCL", riemann="HLL_Toro", precision="fp32c",
                    time="RK2", cfl=0.45, crossings=0.1, n_x=0, n_y=0, steps=0)
    c = dict(kind=kind, scheme="MUSCL", riemann="HLL", precision="fp64_fast", time="SingleStep", cfl=0.4,
             steps=rng.randint(8, 40))
    if kind == "tube":
        n = between(96, 480)
        c.update(n_x=n, n_y=between(24, max(25, n // 2)), scheme=rng.choice(["MUSCL", "MHM", "Godunov"]),
                 riemann=rng.choice(["HLL", "StegerWarming", "HLL_Toro"]),
                 precision=rng.choice(["fp64", "fp64_fast"]), t_end=0.1, cfl=0.4, steps=0)
    elif kind == "quad":
        c.update(n_x=between(33, 900), n_y=between(33, 900), scheme=rng.choice(["MUSCL", "MHM", "Godunov"]),
                 riemann=rng.choice(["HLL", "StegerWarming"]), precision=rng.choice(["fp64", "fp64_fast"]))
    elif kind in ("channel", "host"):
        n = between(250, 2300)
        c.update(n_x=n, n_y=n // 2 + rng.randint(-9, 9), boundary=rng.choice(["IDWBaseGFM", "HBCGFM"]),
                 riemann=rng.choice(["HLL", "HLLC", "StegerWarming"]), cfl=0.45,
                 precision=rng.choice(["fp64", "fp64_fast", "fp64_fast", "fp32c"]), steps=rng.randint(8, 24))
        if kind == "host":
            c.update(precision="fp64_fast", steps=rng.randint(8, 24))
    elif kind == "vortex":
        fp32 = rng.random() < 0.5
        c.update(n_x=between(200, 3000 if fp32 else 1100), scheme=rng.choice(["MUSCL", "MHM"]), riemann="HLL_Toro",
                 precision="fp32c" if fp32 else "fp64_fast", time=rng.choice(["RK2", "RK2", "SingleStep"]), cfl=0.25,
                 steps=rng.randint(4, 10))
        c["n_y"] = c["n_x"]
    else:
        n = between(400, 3500)
        c.update(n_x=n, n_y=n // 2 + rng.randint(-5, 5), riemann="HLL_Toro",
                 precision="fp32c" if n > 1200 else rng.choice(["fp32c", "fp64_fast"]), cfl=0.3,
                 steps=rng.randint(8, 20))
    return c


# ---------------------------------------------------------------- inputs


def _grid(case):
    n_x, n_y = case["n_x"], case["n_y"]
    width = {"tube": 1.0, "quad": 1.0, "channel": 2.0, "host": 2.0, "vortex": 10.0, "obstacles": 4.0}[case["kind"]]
    return plug.Grid(n_x, n_y, 2, 0.0, 0.0, width, width * n_y / n_x)  # square cells


def _boundary(case):
    return {"channel": case.get("boundary"), "host": case.get("boundary"), "obstacles": "CCM"}.get(case["kind"], "Regular")


def _gas(rng, state):
    """`state` with its density and pressure changed by up to a tenth."""
    return (state[0] * rng.uniform(0.9, 1.1), state[1], state[2], state[3] * rng.uniform(0.9, 1.1))


def _fields(case, seed):
    """Level set (N, M) and initial conserved state (N, M, 4), float64 tensors on
    the GPU; cells outside the fluid hold what the reference's Initialize writes."""
    rng = random.Random(seed)
    g = _grid(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dx = (g.hi_x - g.lo_x) / g.n_x
    x = (-dx * g.ng + g.lo_x + dx / 2) + torch.arange(g.M, dtype=torch.float64, device=dev)[None, :] * dx
    y = (-dx * g.ng + g.lo_y + dx / 2) + torch.arange(g.N, dtype=torch.float64, device=dev)[:, None] * dx
    phi = torch.ones((g.N, g.M), dtype=torch.float64, device=dev)

    def conserved(s):
        r, u, v, p = s
        return torch.tensor([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)], dtype=torch.float64,
                            device=dev)

    high, low = (1.0, 0.0, 0.0, 1.0), (0.125, 0.0, 0.0, 0.1)
    if case["kind"] == "tube":
        left = (x < rng.uniform(0.45, 0.55)).expand(g.N, g.M)
        u = torch.where(left[..., None], conserved(_gas(rng, high)), conserved(_gas(rng, low)))
    elif case["kind"] == "quad":
        st = [conserved(_gas(rng, s)) for s in ((1.0, 0.1, 0.3, 1.0), (0.6, -0.1, 0.2, 0.7), (0.9, 0.0, 0.3, 0.9),
                                                (1.1, 0.2, 0.0, 1.1))]
        right, top = x >= rng.uniform(0.4, 0.6), y >= g.hi_y * rng.uniform(0.4, 0.6)
        u = torch.where((top & right)[..., None], st[0], torch.where((top & ~right)[..., None], st[1], torch.where(
            (~top & ~right)[..., None], st[2], st[3])))
    elif case["kind"] in ("channel", "host"):
        th, wid = math.radians(30.0), 0.25
        cx, cy = 0.5 * g.hi_x, 0.5 * g.hi_y
        s = (x - cx) * (-math.sin(th)) + (y - cy) * math.cos(th)
        phi = torch.minimum(s + 0.5 * wid, 0.5 * wid - s)
        a = (x - cx) * math.cos(th) + (y - cy) * math.sin(th)
        u = torch.where((a < rng.uniform(-0.1, 0.1))[..., None], conserved(_gas(rng, high)), conserved(_gas(rng, low)))
        solid = _cell_types(g, phi) == 1
        u = torch.where(solid[..., None], torch.tensor([-1.0, 0.0, 0.0, -1.0], dtype=torch.float64, device=dev), u)
    else:  # vortex
        beta, xc, yc = rng.uniform(4.5, 5.2), rng.uniform(2.0, 8.0), rng.uniform(2.0, 8.0)
        L = g.hi_x
        ex, ey = (x - xc + 0.5 * L) % L - 0.5 * L, (y - yc + 0.5 * L) % L - 0.5 * L
        r2 = ex * ex + ey * ey
        f = torch.exp(0.5 * (1.0 - r2))
        vx, vy = 1.0 - beta / (2 * math.pi) * ey * f, 1.0 + beta / (2 * math.pi) * ex * f
        T = 1.0 - (GAMMA - 1) * beta * beta / (8 * GAMMA * math.pi ** 2) * torch.exp(1.0 - r2)
        r = T ** (1.0 / (GAMMA - 1))
        u = torch.stack([r, r * vx, r * vy, r * T / (GAMMA - 1) + 0.5 * r * (vx * vx + vy * vy)], dim=-1)
    return phi, u.contiguous()


def _bodies(case, seed):
    return [ib.circle(o.xc, o.yc, o.a) if o.kind == "circle" else ib.ellipse(o.xc, o.yc, o.a, o.b, o.theta)
            for o in plug.random_obstacles(seed=seed % (1 << 31), height=_grid(case).hi_y)]


def _requests(case, seed):
    """The stream's requests: sizes from the case, shock and body from the seed."""
    size, rng = random.Random(case["stream"]), random.Random(seed)
    out = []
    for k in range(case["requests"]):
        cells = math.exp(size.uniform(math.log(case["min_cells"]), math.log(case["max_cells"])))
        aspect = size.uniform(1.0, 4.0)
        n_x = max(16, int(round(math.sqrt(cells * aspect))))
        n_y = max(16, int(round(cells / n_x)))
        H, mach = n_y / n_x, rng.uniform(1.5, 4.0)
        out.append(dict(n_x=n_x, n_y=n_y, H=H, mach=mach, r=rng.uniform(0.05, 0.2) * H, xc=rng.uniform(0.15, 0.4),
                        yc=rng.uniform(0.3, 0.7) * H, t_end=case["crossings"] / (mach * math.sqrt(GAMMA))))
    return out


def _case(case):
    g = _grid(case)
    return ib.Case(g.n_x, g.n_y, lo=(0.0, 0.0), hi=(g.hi_x, g.hi_y), gamma=GAMMA, cfl=case["cfl"],
                   t_end=case.get("t_end", FOREVER), max_iter=2 ** 31 - 1, scheme=case["scheme"],
                   riemann=case["riemann"], boundary=_boundary(case),
                   gbc="periodic" if case["kind"] == "vortex" else "walls", precision=case["precision"],
                   time=case["time"])


def _pinned(n, values=None):
    """A page-locked array of n doubles (or of a tensor's values)."""
    a = torch.empty(n, dtype=torch.float64, pin_memory=True)
    if values is not None:
        a.copy_(values.reshape(-1))
    return a


def prepare(case, seed):
    if case["kind"] == "served":
        reqs = _requests(case, seed)
        rho = [_pinned(r["n_x"] * r["n_y"]) for r in reqs]
        made = [ib.request(k, r["n_x"], r["n_y"], (0.0, 0.0), (1.0, r["H"]), r["t_end"],
                           bodies=[ib.circle(r["xc"], r["yc"], r["r"])], x_split=0.1, left=plug.post_shock(r["mach"]),
                           cfl=case["cfl"], boundary="IDWBaseGFM", density_out=b.data_ptr())
                for k, (r, b) in enumerate(zip(reqs, rho))]
        server = ib.Server(scheme=case["scheme"], riemann=case["riemann"], precision=case["precision"],
                           time=case["time"], tile_shape="32x16")
        return dict(kind="served", server=server, requests=made, rho=rho)
    c = _case(case)
    if case["kind"] == "obstacles":
        c.setup_bodies(_bodies(case, seed))
        post = plug.post_shock(random.Random(seed).uniform(2.5, 3.2))
        return dict(kind="obstacles", case=c, steps=case["steps"], post=post, out=_pinned(c.M * c.N * 4))
    phi, u = _fields(case, seed)
    c.setup_geometry(phi.cpu().numpy())
    if case["kind"] == "host":
        return dict(kind="host", case=c, steps=case["steps"], u0=_pinned(u.numel(), u), u=_pinned(u.numel()))
    return dict(kind="run" if case["steps"] == 0 else "advance", case=c, steps=case["steps"], u0=_pinned(u.numel(), u),
                out=_pinned(c.M * c.N * 4))


# ---------------------------------------------------------------- one pass


def _loop_scalars(p):
    return {k: p[k] for k in ("iter", "now_t", "dt", "mass")}


def run(state):
    kind = state["kind"]
    if kind == "served":
        server = state["server"]
        for r in state["requests"]:
            server.submit(r)
        server.run()
        done = sorted(server.poll(), key=lambda r: r["id"])
        return {"iter": [r["iter"] for r in done], "now_t": [r["now_t"] for r in done],
                "rho": state["rho"]}
    c = state["case"]
    if kind == "host":
        c.set_state_ptr(state["u0"].data_ptr())
        u = state["u"]
        c.get_state_ptr(u.data_ptr())  # the walls' ghost cells filled
        for _ in range(state["steps"]):
            p = c.step_host_ptr(u.data_ptr(), u.data_ptr())
        return {"state": u, "loop": _loop_scalars(p)}
    if kind == "obstacles":
        c.init_x_split(0.5, state["post"], (1.0, 0.0, 0.0, 1.0))
    else:
        c.set_state_ptr(state["u0"].data_ptr())
    if kind == "run":
        p = c.run()
    else:
        c.advance(state["steps"])
        p = c.progress()
    c.get_state_ptr(state["out"].data_ptr())
    return {"state": state["out"], "loop": _loop_scalars(p)}


# ---------------------------------------------------------------- what a pass cannot do without

# floating-point operations of one face (reconstruction, two primitive states,
# wave speeds, flux) and of one cell (update, CFL maxima, mass); an MHM face
# evaluates two more fluxes
FACE_FLOPS, MHM_FLOPS, CELL_FLOPS = 110, 50, 45


def work(case):
    stages = 2 if case["time"] == "RK2" else 1
    flops = 2 * (FACE_FLOPS + (MHM_FLOPS if case["scheme"] == "MHM" else 0)) + CELL_FLOPS
    # per fluid cell and step: each stage reads and writes the state (32 B
    # each) and reads the cell type; RK2's second stage reads the first state too
    per_step = 65 * stages + (32 if stages == 2 else 0)
    if case["kind"] == "served":
        b = f = 0.0
        for r in _requests(case, 0):
            n = r["n_x"] * r["n_y"]
            rho2, u2, _, p2 = plug.post_shock(2.75)
            steps = math.ceil(r["t_end"] / (case["cfl"] / r["n_x"]) * (u2 + math.sqrt(GAMMA * p2 / rho2)))
            b += n * (per_step * steps + 40)
            f += n * flops * stages * steps
        return {"bytes": b, "flops": f}
    cells = case["n_x"] * case["n_y"]
    fluid = cells * {"channel": 0.25, "host": 0.25, "obstacles": 0.93}.get(case["kind"], 1.0)
    steps = case["steps"]
    if steps == 0:  # to t_end: the fastest wave of the tube is about 2.2
        steps = math.ceil(case["t_end"] * 2.2 * case["n_x"] / case["cfl"])
    moved = 32 * cells * (1 if case["kind"] == "obstacles" else 2)  # the state in and out
    if case["kind"] == "host":
        moved = 64 * fluid * steps
    return {"bytes": float(fluid * per_step * steps + moved), "flops": float(fluid * flops * stages * steps)}


# ---------------------------------------------------------------- the same in plain 64-bit torch


def _cell_types(g, phi):
    """0 fluid, 1 solid, 2 ghost (a solid cell within two of the fluid along x or y) and the domain's ring."""
    ng, t = g.ng, torch.full_like(phi, 2.0)
    inside = (slice(ng, ng + g.n_y), slice(ng, ng + g.n_x))
    fluid = torch.zeros_like(phi, dtype=torch.bool)
    fluid[inside] = phi[inside] >= 0
    near = torch.zeros_like(fluid)
    for k in range(1, ng + 1):
        near[:, k:] |= fluid[:, :-k]
        near[:, :-k] |= fluid[:, k:]
        near[k:] |= fluid[:-k]
        near[:-k] |= fluid[k:]
    t[inside] = torch.where(fluid, 0.0, torch.where(near, 2.0, 1.0))[inside].to(t.dtype)
    return t


class _Walls:
    """Ghost cells of the immersed walls: image points, brackets, inverse-distance weights."""

    def __init__(self, g, phi, types, boundary):
        ng, dx = g.ng, (g.hi_x - g.lo_x) / g.n_x
        inner = torch.zeros_like(types, dtype=torch.bool)
        inner[ng:ng + g.n_y, ng:ng + g.n_x] = True
        self.j, self.i = torch.nonzero(inner & (types == 2), as_tuple=True)
        self.mixed = boundary != "IDWBaseGFM"
        dev = phi.device
        X = (-dx * ng + g.lo_x + dx / 2) + torch.arange(g.M, dtype=torch.float64, device=dev) * dx
        Y = (-dx * ng + g.lo_y + dx / 2) + torch.arange(g.N, dtype=torch.float64, device=dev) * dx
        self.nx = (phi[self.j, self.i + 1] - phi[self.j, self.i - 1]) / (X[self.i + 1] - X[self.i - 1])
        self.ny = (phi[self.j + 1, self.i] - phi[self.j - 1, self.i]) / (Y[self.j + 1] - Y[self.j - 1])
        d = phi[self.j, self.i].abs()
        self.d, self.delta = d, math.sqrt(2.0) * dx / 2
        self.mirror = d > self.delta
        reach = [2 * d] if not self.mixed else [torch.where(self.mirror, 2 * d, d + self.delta),
                                                torch.where(self.mirror, 2 * d, d + 2 * self.delta)]
        self.points = []
        for r in reach:
            xm, ym = X[self.i] + self.nx * r, Y[self.j] + self.ny * r
            bi = (torch.searchsorted(X, xm, right=True) - 1).clamp(0, g.M - 2)
            bj = (torch.searchsorted(Y, ym, right=True) - 1).clamp(0, g.N - 2)
            corner = [(bj, bi), (bj + 1, bi), (bj + 1, bi + 1), (bj, bi + 1)]
            w = []
            for cj, ci in corner:
                ok = (types[cj, ci] != 1) if self.mixed else (types[cj, ci] < 1)
                w.append(torch.where(ok, 1 / torch.sqrt((X[ci] - xm) ** 2 + (Y[cj] - ym) ** 2), torch.zeros_like(xm)))
            self.points.append((corner, w))

    def _average(self, S, point):
        corner, w = point
        total, out = sum(w), [0.0] * 4
        for (cj, ci), a in zip(corner, w):
            r, u, v, p = _primitive(S[:, cj, ci])
            out = [o + a * q for o, q in zip(out, (r, u, v, p))]
        return [o / total for o in out]

    def fill(self, S, U):
        nx, ny = self.nx, self.ny
        r, u, v, p = self._average(S, self.points[0])
        un, ut = u * nx + v * ny, u * ny - v * nx
        if self.mixed:
            r2, u2, v2, p2 = self._average(S, self.points[1])
            un2, ut2 = u2 * nx + v2 * ny, u2 * ny - v2 * nx
            e = self.delta

            def mix(a, b):
                q = (a * ((e + e) ** 2 - self.d ** 2) - b * (e * e - self.d ** 2)) / (e * e + 2 * e * e)
                return torch.where(self.mirror, a, q)

            r, p, ut, un = mix(r, r2), mix(p, p2), mix(ut, ut2), mix(un, un2)
        un = -un
        u, v = un * nx + ut * ny, un * ny - ut * nx
        U[:, self.j, self.i] = torch.stack([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)])


def _primitive(U):
    u, v = U[1] / U[0], U[2] / U[0]
    return U[0], u, v, (GAMMA - 1) * (U[3] - 0.5 * U[0] * (u * u + v * v))


def _flux(U, n):
    r, u, v, p = _primitive(U)
    q = u if n == 1 else v
    F = torch.stack([r * q, r * u * q, r * v * q, (U[3] + p) * q])
    F[n] += p
    return F


def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() > b.abs(), b, a), torch.zeros_like(a))


def _internal(U):
    return U[3] - 0.5 * (U[1] * U[1] + U[2] * U[2]) / U[0]


def _riemann(L, R, riemann, n):
    """Face flux and, for the reference's HLL in y, where its solver leaves the flux slot alone."""
    rl, ul, vl, pl = _primitive(L)
    rr, ur, vr, pr = _primitive(R)
    ql, qr = (ul, ur) if n == 1 else (vl, vr)
    al, ar = torch.sqrt(GAMMA * pl / rl), torch.sqrt(GAMMA * pr / rr)
    none = torch.zeros_like(rl, dtype=torch.bool)
    if riemann == "StegerWarming":
        F = 0.0
        for U, r, u, v, q, p, a, sign in ((L, rl, ul, vl, ql, pl, al, 1.0), (R, rr, ur, vr, qr, pr, ar, -1.0)):
            l1, l3, l4 = (0.5 * (s + sign * torch.sqrt(s * s + 1e-12)) for s in (q, q - a, q + a))
            h = p / (GAMMA - 1) / r + 0.5 * (u * u + v * v) + p / r
            t = 2 * (GAMMA - 1) * l1 + l3 + l4
            out = [t, u * t, v * t, (GAMMA - 1) * (u * u + v * v) * l1 + (h - a * q) * l3 + (h + a * q) * l4]
            out[n] = 2 * (GAMMA - 1) * q * l1 + (q - a) * l3 + (q + a) * l4
            F = F + r / (2 * GAMMA) * torch.stack(out)
        return F, none
    ps = 0.5 * (pl + pr) + 0.125 * (ql - qr) * (rl + rr) * (al + ar)
    c1, c2 = (GAMMA + 1) / (2 * GAMMA), (GAMMA - 1) / (2 * GAMMA)
    if riemann == "HLL_Toro":
        ps = ps.clamp(min=0.0)
        kl = torch.where(ps > pl, torch.sqrt(c1 * ps / pl + c2), torch.ones_like(ps))
        kr = torch.where(ps > pr, torch.sqrt(c1 * ps / pr + c2), torch.ones_like(ps))
    else:
        kl, kr = torch.sqrt(c1 * ps / pl + c2), torch.sqrt(c1 * ps / pr + c2)
    sl, sr = ql - al * kl, qr + ar * kr
    FL, FR = _flux(L, n), _flux(R, n)
    F = torch.where(sl >= 0, FL, torch.where(sr <= 0, FR, (sr * FL - sl * FR + sr * sl * (R - L)) / (sr - sl)))
    return F, (sl >= 0) if n == 2 and riemann in ("HLL", "HLLC") else none


def _faces(U, case, dt, h, n):
    """Fluxes of the faces between cells k and k + 1, k = 1 ... length - 3, along x (n = 1) or y (n = 2)."""
    if n == 2:
        U = U.transpose(1, 2)
    c0, c1, c2, c3 = (U[:, :, k:U.shape[2] - 3 + k] for k in range(4))
    L, R = c1, c2
    if case["scheme"] != "Godunov":
        d = c2 - c1
        L, R = c1 + 0.5 * _minmod(c1 - c0, d), c2 - 0.5 * _minmod(c3 - c2, d)
        if case["scheme"] == "MHM":
            s = 0.5 * (_flux(L, n) - _flux(R, n)) * dt / h
            L, R = L + s, R + s
        if case["riemann"] == "HLL_Toro":
            def sound(V):
                return (V[0] > 0) & (_internal(V) > 1e-6 * V[3].abs())
            bad = sound(c1) & sound(c2) & ~(sound(L) & sound(R))
            L, R = torch.where(bad, c1, L), torch.where(bad, c2, R)
    F, kept = _riemann(L, R, case["riemann"], n)
    return (F, kept) if n == 1 else (F.transpose(1, 2), kept.transpose(0, 1))


class _Plain:
    """The time loop on whole arrays (4, N, M)."""

    def __init__(self, g, case, boundary, gbc, phi, u0):
        self.g, self.case, self.gbc, self.boundary = g, case, gbc, boundary
        self.dx, self.dy = (g.hi_x - g.lo_x) / g.n_x, (g.hi_y - g.lo_y) / g.n_y
        types = _cell_types(g, phi)
        self.fluid = types == 0
        self.walls = _Walls(g, phi, types, boundary) if boundary != "Regular" else None
        self.U = u0.permute(2, 0, 1).clone()
        self.first = self.U.clone()
        if self.walls:
            self.walls.fill(self.first, self.U)
        self.t, self.iter = 0.0, 0
        self._dt()

    def _dt(self):
        r, u, v, p = _primitive(self.U)
        a, u, v = (torch.where(self.fluid, q, torch.zeros_like(q)).max() for q in (torch.sqrt(GAMMA * p / r), u.abs(),
                                                                                      v.abs()))
        self.dt = float(self.case["cfl"] * self.dx / (a + torch.maximum(u, v)))

    def _rate(self, U):
        ng, g, dt = self.g.ng, self.g, self.dt
        F, _ = _faces(U, self.case, dt, self.dx, 1)
        G, kept = _faces(U, self.case, dt, self.dy, 2)
        # x faces of columns 1 ... M - 3, y faces of rows 1 ... N - 3 (two ghost layers)
        cols, rows = slice(ng, ng + g.n_x), slice(ng, ng + g.n_y)
        G = torch.where(kept[:, cols], F[:, 1:g.N - 2, 1:], G[:, :, cols])
        d = torch.zeros_like(U)
        d[:, rows, cols] = (F[:, rows, 1:] - F[:, rows, :-1]) / self.dx + (G[:, 1:] - G[:, :-1]) / self.dy
        return d

    def _stage(self, U, old):
        """The state after Boundary and Global_Boundary: `U` holds the new fluid cells, `old` the state before."""
        g, ng = self.g, self.g.ng
        S = torch.where(self.fluid, U, old)
        ring = self.first if self.boundary == "Regular" else old
        S[:, :ng], S[:, ng + g.n_y:] = ring[:, :ng], ring[:, ng + g.n_y:]
        S[:, :, :ng], S[:, :, ng + g.n_x:] = ring[:, :, :ng], ring[:, :, ng + g.n_x:]
        V = torch.where(self.fluid, U, old)
        if self.walls:
            self.walls.fill(S, V)
        top, right = ng + g.n_y, ng + g.n_x
        if self.gbc == "periodic":
            V[:, :ng], V[:, top:] = V[:, g.n_y:top], V[:, ng:2 * ng]
            V[:, :, :ng], V[:, :, right:] = V[:, :, g.n_x:right], V[:, :, ng:2 * ng]
            return V
        for k in range(ng):
            V[:, k], V[:, top + k] = S[:, 2 * ng - 1], S[:, top - 1]
            V[2, k], V[2, top + k] = -S[2, 2 * ng - 1 - k], -S[2, top - 1 - k]
        for k in range(ng):
            V[:, :, k], V[:, :, right + k] = S[:, :, ng], S[:, :, right - 1]
        return V

    def _floor(self, U):
        if self.case["riemann"] != "HLL_Toro":
            return U
        e, f = _internal(U), 1e-5 * U[3].abs()
        U[3] = torch.where((U[0] > 0) & (e < f), (U[3] - e) + f, U[3])
        return U

    def step(self):
        U = self.U
        V = self._floor(U - self.dt * self._rate(U))
        if self.case["time"] == "RK2":
            V = self._stage(V, U)
            W = 0.5 * (U + self._floor(V - self.dt * self._rate(V)))
            self.U = self._stage(W, V)
        else:
            self.U = self._stage(V, U)
        self._dt()
        self.t += self.dt
        self.iter += 1

    def loop(self):
        mass = float(torch.where(self.fluid, self.U[0], torch.zeros_like(self.U[0])).sum()) * self.dx * self.dy
        return {"iter": self.iter, "now_t": self.t, "dt": self.dt, "mass": mass}


def exact(case, seed):
    if case["kind"] == "obstacles":
        return None  # the cut-cell geometry and its mixing lists have no short form on whole arrays
    if case["kind"] == "served":
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        its, ts, rho = [], [], []
        for r in _requests(case, seed):
            g = plug.Grid(r["n_x"], r["n_y"], 2, 0.0, 0.0, 1.0, r["H"])
            dx = 1.0 / g.n_x
            x = (-2 * dx + dx / 2) + torch.arange(g.M, dtype=torch.float64, device=dev)[None, :] * dx
            y = (-2 * dx + dx / 2) + torch.arange(g.N, dtype=torch.float64, device=dev)[:, None] * dx
            phi = torch.sqrt((x - r["xc"]) ** 2 + (y - r["yc"]) ** 2) - r["r"]
            two = []
            for d, u, v, p in (plug.post_shock(r["mach"]), (1.0, 0.0, 0.0, 1.0)):
                two.append(torch.tensor([d, d * u, d * v, p / (GAMMA - 1) + 0.5 * d * (u * u + v * v)],
                                        dtype=torch.float64, device=dev))
            u0 = torch.where((x < 0.1).expand(g.N, g.M)[..., None], two[0], two[1])
            u0[_cell_types(g, phi) == 1] = torch.tensor([-1.0, 0.0, 0.0, -1.0], dtype=torch.float64, device=dev)
            s = _Plain(g, case, "IDWBaseGFM", "walls", phi, u0)
            while s.t < r["t_end"]:
                s.step()
            its.append(s.iter)
            ts.append(s.t)
            rho.append(s.U[0, 2:-2, 2:-2].reshape(-1))
        return {"iter": its, "now_t": ts, "rho": rho}
    phi, u = _fields(case, seed)
    s = _Plain(_grid(case), case, _boundary(case), "periodic" if case["kind"] == "vortex" else "walls", phi, u)
    while s.t < case["t_end"] if case["steps"] == 0 else s.iter < case["steps"]:
        s.step()
    return {"state": s.U.permute(1, 2, 0).reshape(-1), "loop": s.loop()}
