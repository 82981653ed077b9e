"""Timing cases of the solver: what a user's program has it do, through ausm's public classes.

Kinds of case:
  frame   n RK3 steps of one solve (dt held, as the reference's frame loop), then the surface
          forces and the state read back: Solver.step / forces / state
  batch   a chunk of steps of many solves together, residual norms, states: Batch.step / residual_l2
  serve   a burst of requests to a running server, served to their step limit: Server.submit / drain / poll
  grid    prepareGrid, an O-grid from its boundary curves: Solver.prepare_grid / vertices

Sizes are this repository's own: the smallest golden grids, the batch and served ranges (128 x 96 ..
1024 x 768), the reference's default 510 x 381 and its README scale 512 x 384, and the large
4096 x 3072 workload.  The state of a frame or batch starts as a freestream with smooth disturbances
of a few per cent, so that every cell has gradients, and goes on from pass to pass as in a run.

exact() restates the path in 64 bits with torch alone (Grid, Flow below).
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = str(Path(__file__).resolve().parent.parent / "ausm-webgpu_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import ausm  # noqa: E402

SCHEMES = ("SLAU2", "SLAU", "AUSM+-up")
ENGINES = ("fused", "reference", "f64")
NACA = (12, 15, 18, 1412, 2312, 2412, 2415, 3510, 4412, 4415, 5410, 6409)
FLOPS = 500  # floating operations of one cell and RK stage: two faces, primitives, residual, combination


def listed():
    return [
        # the smallest call: one step and a look at the state, as an interactive host does
        dict(name="frame_64x33_step1", kind="frame", engine="fused", M=64, N=33, scheme="SLAU2", muscl=1, mach=0.8,
             n=1, sweeps=100),
        # a short frame of the smallest batch-range grid, one solve alone
        dict(name="frame_128x96_ausmup", kind="frame", engine="fused", M=128, N=96, scheme="AUSM+-up", muscl=1,
             mach=2.0, n=20, sweeps=200),
        # first-order faces on an odd grid: the robust start-up setting
        dict(name="frame_257x131_slau_first_order", kind="frame", engine="fused", M=257, N=131, scheme="SLAU",
             muscl=0, mach=1.5, n=50, sweeps=200),
        # the README-scale grid in frames of 100 steps
        dict(name="frame_512x384_slau2", kind="frame", engine="fused", M=512, N=384, scheme="SLAU2", muscl=1,
             mach=0.8, n=100, sweeps=200),
        # an odd grid of a million cells, hypersonic
        dict(name="frame_1155x867_slau", kind="frame", engine="fused", M=1155, N=867, scheme="SLAU", muscl=1,
             mach=6.0, n=50, sweeps=200),
        # the large precision-study grid
        dict(name="frame_4096x3072_slau2", kind="frame", engine="fused", M=4096, N=3072, scheme="SLAU2", muscl=1,
             mach=6.0, n=50, sweeps=200),
        # uneven solves stepped together (parameter sweeps)
        dict(name="batch_12_uneven", kind="batch", members=12, cells_lo=128 * 96, cells_hi=1024 * 768, n=100,
             sweeps=100),
        # a burst of requests to a running server
        dict(name="serve_6_requests", kind="serve", requests=6, cells_lo=64 * 48, cells_hi=320 * 240, steps=200,
             sweeps=200),
        # the reference's own generator at its default size
        dict(name="grid_jacobi_510x381", kind="grid", method="jacobi", M=510, N=381, sweeps=2000),
        # the FP64 generator on a large batch-range grid
        dict(name="grid_multicolor_1024x768", kind="grid", method="multicolor", M=1024, N=768, sweeps=200),
        # the precision reference run beside an FP32 solve
        dict(name="frame_512x384_f64", kind="frame", engine="f64", M=512, N=384, scheme="SLAU2", muscl=1, mach=0.8,
             n=10, sweeps=200),
        # the engine that reproduces the reference bit for bit, at the reference's default size
        dict(name="frame_510x381_reference", kind="frame", engine="reference", M=510, N=381, scheme="AUSM+-up",
             muscl=1, mach=2.0, n=20, sweeps=200),
    ]


def draw(rng):
    def size(lo, hi):  # cells log-uniform, aspect 4:3, any parity
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        M = max(32, int(math.sqrt(cells * 4.0 / 3.0)) + rng.randrange(0, 2))
        return M, max(16, int(cells / M) + rng.randrange(0, 2))

    kind = rng.choice(("frame", "frame", "frame", "frame", "batch", "serve", "jacobi", "multicolor", "f64", "reference"))
    if kind == "batch":
        return dict(kind="batch", members=rng.randrange(2, 13), cells_lo=rng.randrange(3000, 13000),
                    cells_hi=rng.randrange(40000, 1024 * 768), n=rng.randrange(20, 101), sweeps=100)
    if kind == "serve":
        return dict(kind="serve", requests=rng.randrange(1, 7), cells_lo=64 * 48, cells_hi=rng.randrange(8000, 320 * 240),
                    steps=100 * rng.randrange(1, 3), sweeps=200)
    if kind == "jacobi":
        M, N = size(2000, 400000)
        return dict(kind="grid", method="jacobi", M=M, N=N, sweeps=rng.randrange(200, 2001))
    if kind == "multicolor":
        M, N = size(2000, 3000000)
        return dict(kind="grid", method="multicolor", M=M, N=N, sweeps=rng.randrange(100, 201))
    mach = rng.choice((0.5, 0.8, 1.5, 2.0, 3.0, 6.0))
    out = dict(kind="frame", engine="fused", scheme=rng.choice(SCHEMES), muscl=int(rng.random() < 0.85), mach=mach)
    if kind == "frame":
        out["M"], out["N"] = size(2000, 12000000)
        out["n"] = rng.randrange(1, 51)
    else:
        out["engine"] = kind
        out["M"], out["N"] = size(2000, 300000)
        out["n"] = rng.randrange(1, 21)
    out["sweeps"] = 100
    return out


# ---- inputs ----
def shape(rng, case):
    """The airfoil, angle of attack and Mach number that a seed gives a solve."""
    return dict(naca=NACA[rng.randint(len(NACA))], aoa=float(rng.uniform(-2.0, 4.0)),
                mach=float(case.get("mach", 1.0) * rng.uniform(0.95, 1.05)))


def far_radius(case):
    return 40.0 if case["M"] * case["N"] > 4000000 else 20.0


def disturbed_state(M, N, mach, aoa, rng):
    """float32 (N+3, M, 4) state in the reference layout: the freestream with smooth
    disturbances (six Fourier modes per primitive variable)."""
    dev = "cuda"
    i = torch.arange(M, device=dev, dtype=torch.float64) * (2 * math.pi / M)
    j = torch.arange(N + 3, device=dev, dtype=torch.float64) * (2 * math.pi / (N + 3))
    a = math.radians(aoa)
    prim = []
    for base, amp in ((1.0, 0.01), (mach * math.cos(a), 0.01), (mach * math.sin(a), 0.01), (1.0 / 1.4, 0.007)):
        f = torch.full((N + 3, M), base, device=dev, dtype=torch.float64)
        for _ in range(6):
            kx, ky, ph = int(rng.randint(0, 6)), int(rng.randint(0, 4)), float(rng.uniform(0, 2 * math.pi))
            f += amp * rng.uniform(0.2, 1.0) * torch.cos(kx * i[None, :] + ky * j[:, None] + ph)
        prim.append(f)
    rho, u, v, p = prim
    return torch.stack((rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)), dim=-1).float().cpu().numpy()


def sizes_of(case, count):
    """Grid sizes (cells log-uniform, aspect 4:3) and schemes of a case's solves, whatever the seed."""
    rng, out = np.random.RandomState(20261203), []
    for _ in range(count):
        cells = math.exp(rng.uniform(math.log(case["cells_lo"]), math.log(case["cells_hi"])))
        M = max(32, int(math.sqrt(cells * 4.0 / 3.0)))
        out.append(dict(M=M, N=max(24, int(cells / M)), sweeps=case["sweeps"], scheme=SCHEMES[rng.randint(3)], muscl=1))
    return out


def batch_members(case, rng):
    out = []
    for d in sizes_of(case, case["members"]):
        d["mach"] = float(rng.uniform(0.3, 3.0))
        d.update(shape(rng, d))
        out.append(d)
    return out


def requests_of(case, rng):
    return [dict(d, naca=NACA[rng.randint(len(NACA))], mach=float(rng.uniform(0.3, 3.0)),
                 aoa=float(rng.uniform(-2.0, 4.0))) for d in sizes_of(case, case["requests"])]


def solver_of(d, engine="fused"):
    """A Solver with d's grid, parameters and engine, without a state."""
    s = ausm.Solver(d["M"], d["N"])
    s.set_body_naca4(d["naca"], 0.5, 0.0)
    s.set_outer_circle(far_radius(d))
    s.set_radial_stretch(1e-3)
    s.generate_grid(d["sweeps"], "multicolor")
    if engine == "reference":  # that engine's metrics are made of the float32 vertices
        s.set_vertices(s.vertices())
    s.set_params(gamma=1.4, in_rho=1.0, in_pressure=1.0 / 1.4, mach=d["mach"], aoa_deg=d["aoa"], K_p=0.0, K_u=0.75,
                 cfl=0.5, maxdt=math.inf, muscl=d["muscl"], scheme=d["scheme"], ramp=0.0)
    if engine != "fused":
        s.set_engine(engine)
    return s


def pinned(shape_):
    """The buffer that a program reads states into, page-locked as its transfers want it."""
    return torch.empty(shape_, dtype=torch.float32, pin_memory=True).numpy()


def prepare(case, seed):
    rng = np.random.RandomState(seed % (1 << 31))
    if case["kind"] == "frame":
        d = dict(case, **shape(rng, case))
        s = solver_of(d, case["engine"])
        s.set_state(disturbed_state(d["M"], d["N"], d["mach"], d["aoa"], rng))
        return dict(case=case, s=s, q=pinned((d["N"] + 3, d["M"], 4)))
    if case["kind"] == "batch":
        b, sol, q = ausm.Batch(), [], []
        for d in batch_members(case, rng):
            s = solver_of(d)
            s.set_state(disturbed_state(d["M"], d["N"], d["mach"], d["aoa"], rng))
            b.add(s)
            sol.append(s)
            q.append(pinned((d["N"] + 3, d["M"], 4)))
        return dict(case=case, b=b, sol=sol, q=q)
    if case["kind"] == "serve":
        srv = ausm.Server(max_active=16, chunk_steps=100)
        srv.start()
        return dict(case=case, srv=srv, reqs=requests_of(case, rng))
    d = dict(case, **shape(rng, case))
    s = ausm.Solver(d["M"], d["N"])
    s.set_body_naca4(d["naca"], 0.5, 0.0)
    s.set_outer_circle(20.0)
    s.set_radial_stretch(1e-3)
    return dict(case=case, s=s)


def run(st):
    case = st["case"]
    if case["kind"] == "frame":
        s = st["s"]
        dt = s.step(case["n"])
        f = s.forces()
        wide = case["engine"] == "f64"
        return dict(dt=dt, forces=np.array([f[k] for k in ("Fx", "Fy", "Cl", "Cd")], np.float64 if wide else np.float32),
                    state=s.state_f64() if wide else s.state(out=st["q"]))
    if case["kind"] == "batch":
        dt_wave = st["b"].step(case["n"])
        l2 = st["b"].residual_l2()
        # norms of an FP32 residual: 32 bits of the double hold it
        return dict(dt_wave=dt_wave, l2=l2.astype(np.float32), states=[s.state(out=q) for s, q in zip(st["sol"], st["q"])])
    if case["kind"] == "serve":
        srv = st["srv"]
        ids = [srv.submit(ausm.make_request(r["M"], r["N"], naca4=r["naca"], grid_iters=r["sweeps"], residual_drop=0.0,
                                            max_steps=case["steps"], mach=r["mach"], aoa_deg=r["aoa"],
                                            scheme=r["scheme"])) for r in st["reqs"]]
        srv.drain()
        out = []
        for i in ids:
            d = srv.poll(i)
            # coefficients of an FP32 state: 32 bits of the double hold them
            out.append(dict(steps=d["steps"], stop=d["stop"], Cp=d["Cp"].astype(np.float32),
                            forces=np.array([d[k] for k in ("Fx", "Fy", "Cl", "Cd")], np.float32)))
        return out
    s = st["s"]
    done = s.prepare_grid(case["sweeps"], case["method"])
    return dict(done=done, vertices=s.vertices())


def work(case):
    """Bytes: the state and vertices in once and the state out once (a grid: its vertices out);
    operations: those of every cell, stage and step, or of every vertex and sweep."""
    rng = np.random.RandomState(0)
    if case["kind"] == "grid":
        v = case["M"] * (case["N"] + 1)
        return dict(bytes=8.0 * v, flops=60.0 * v * case["sweeps"])
    if case["kind"] == "frame":
        width = 2 if case["engine"] == "f64" else 1
        solves, n, sweeps = [case], case["n"], 0
    elif case["kind"] == "batch":
        width, solves, n, sweeps = 1, batch_members(case, rng), case["n"], 0
    else:
        width, solves, n, sweeps = 1, requests_of(case, rng), case["steps"], case["sweeps"]
    cells = sum(float(d["M"]) * d["N"] for d in solves)
    return dict(bytes=width * 40.0 * cells, flops=cells * (3.0 * FLOPS * n + 60.0 * sweeps))


# ---- the same in 64 bits, with torch alone ----
def naca4_points(M, digits):
    """M body points of a NACA 4-digit airfoil of unit chord centred at the origin, closed trailing edge."""
    t = np.arange(M) / (M / 2.0)
    s = np.where(t <= 1, np.abs(1 - t), np.abs(t - 1)) ** (7.0 / 5.0)
    thick, m, p = digits % 100 / 100.0, (digits // 1000) / 100.0, (digits // 100) % 10 / 10.0
    half = 5 * thick * (0.2969 * np.sqrt(s) - 0.126 * s - 0.3516 * s * s + 0.2843 * s ** 3 - 0.1036 * s ** 4)
    if m > 0:
        k = np.where(s < p, m / (p * p), m / ((1 - p) * (1 - p)))
        camber = k * np.where(s < p, 2 * p * s - s * s, (1 - 2 * p) + 2 * p * s - s * s)
        slope = k * (2 * p - 2 * s)
    else:
        camber, slope = np.zeros(M), np.zeros(M)
    cx, cy = half * -np.sin(np.arctan(slope)), half / np.sqrt(1 + slope * slope)
    up = np.where(t <= 1, 1.0, -1.0)
    return np.stack((s - 0.5 + up * cx, camber + up * cy), axis=-1)


class Grid:
    """O-grid vertices x, y (N+1, M) in 64 bits."""

    def __init__(self, M, N, digits, radius, first, f32_ends):
        self.M, self.N = M, N
        body = naca4_points(M, digits)
        th = np.arange(M) / M * (2 * math.pi)
        outer = np.stack((radius * np.cos(th), radius * np.sin(th)), axis=-1)
        if f32_ends:  # the FP32 generator is given its boundary curves in float32
            body, outer = body.astype(np.float32).astype(np.float64), outer.astype(np.float32).astype(np.float64)
        h = first / np.hypot(*(outer - body).T)
        lo, hi = np.full(M, 1.0 + 1e-12), np.full(M, 2.0)
        small = h * N >= 1.0
        lo[small], hi[small] = 1e-6, 1.0 - 1e-12
        with np.errstate(over="ignore"):
            for _ in range(200):
                q = 0.5 * (lo + hi)
                up = (h * (q ** N - 1) / (q - 1) > 1.0) == ~small
                hi, lo = np.where(up, q, hi), np.where(up, lo, q)
        q = torch.tensor(0.5 * (lo + hi), device="cuda")
        h, j = torch.tensor(h, device="cuda"), torch.arange(N + 1, device="cuda", dtype=torch.float64)
        t = h * (q[None, :] ** j[:, None] - 1) / (q - 1)
        t[0], t[N] = 0.0, 1.0
        body, outer = (torch.tensor(a, device="cuda") for a in (body, outer))
        self.x, self.y = (body[:, k] * (1 - t) + outer[:, k] * t for k in (0, 1))

    def moved(self, rows, cols):
        """New positions of the interior vertices rows x cols (index tensors) by one TTM update."""
        lf, rt = (cols - 1) % self.M, (cols + 1) % self.M

        def at(a, r, c):
            return a[r[:, None], c[None, :]]
        L, R, D, U, DL, DR, UL, UR = ([at(a, rows + dj, c) for a in (self.x, self.y)] for dj, c in (
            (0, lf), (0, rt), (-1, cols), (1, cols), (-1, lf), (-1, rt), (1, lf), (1, rt)))
        xi, et = [0.5 * (b - a) for a, b in zip(L, R)], [0.5 * (b - a) for a, b in zip(D, U)]
        xe = [0.25 * (a + b - c - d) for a, b, c, d in zip(UR, DL, UL, DR)]
        al, ga, be = et[0] ** 2 + et[1] ** 2, xi[0] ** 2 + xi[1] ** 2, xi[0] * et[0] + xi[1] * et[1]
        new = [(al * (L[k] + R[k]) + ga * (D[k] + U[k]) - 2 * be * xe[k]) / (2 * (al + ga)) for k in (0, 1)]
        turned = xi[0] * et[1] - xi[1] * et[0] < 0
        return [torch.where(turned, n, at(a, rows, cols)) for n, a in zip(new, (self.x, self.y))]

    def jacobi(self, sweeps):
        rows, cols = torch.arange(1, self.N, device="cuda"), torch.arange(self.M, device="cuda")
        for _ in range(sweeps):
            x, y = self.moved(rows, cols)
            self.x[1:-1], self.y[1:-1] = x, y

    def multicolor(self, sweeps):
        even = self.M - self.M % 2
        groups = [torch.arange(c, even, 2, device="cuda") for c in (0, 1)]
        if self.M % 2:  # the odd column at the seam has colours of its own
            groups.append(torch.tensor([self.M - 1], device="cuda"))
        rows = [torch.arange(2, self.N, 2, device="cuda"), torch.arange(1, self.N, 2, device="cuda")]
        for _ in range(sweeps):
            for cols in groups:
                for r in rows:
                    if len(r):
                        x, y = self.moved(r, cols)
                        self.x[r[:, None], cols[None, :]], self.y[r[:, None], cols[None, :]] = x, y

    def vertices(self):
        return torch.stack((self.x, self.y), dim=-1)

    def rounded(self):
        self.x, self.y = self.x.float().double(), self.y.float().double()


class Flow:
    """The explicit step in 64 bits: q (4, N, M) conserved."""

    def __init__(self, grid, mach, aoa, scheme, muscl):
        self.g, self.scheme, self.muscl, self.gam = grid, scheme, muscl, 1.4
        x, y = grid.x, grid.y
        xr, yr = x.roll(-1, 1), y.roll(-1, 1)
        ux, uy, tx, ty = x[1:] - x[:-1], y[1:] - y[:-1], x - xr, y - yr
        self.li, self.lj = torch.hypot(ux, uy), torch.hypot(tx, ty)
        self.ni, self.nj = (-uy / self.li, ux / self.li), (-ty / self.lj, tx / self.lj)
        self.A = 0.5 * ((xr[1:] - x[:-1]) * (y[1:] - yr[:-1]) - (x[1:] - xr[:-1]) * (yr[1:] - y[:-1])).abs()
        self.W = (self.li + self.li.roll(-1, 1) + self.lj[1:] + self.lj[:-1]) / (2 * self.A)
        a = math.radians(aoa)
        self.u, self.v = mach * math.cos(a), mach * math.sin(a)  # a_inf = 1
        self.pin = 1.0 / 1.4
        self.instate = torch.tensor([1.0, self.u, self.v, self.pin / 0.4 + 0.5 * mach * mach], device="cuda",
                                    dtype=torch.float64)

    def freestream(self):
        self.q = self.instate[:, None, None].expand(4, self.g.N, self.g.M).contiguous()

    def prim(self, q):
        u, v = q[1] / q[0], q[2] / q[0]
        p = ((q[3] - 0.5 * q[0] * (u * u + v * v)) * 0.4).clamp(min=1e-7)
        return torch.stack((q[0], u, v, p))

    def ghosts(self, q):
        """Conserved wall ghost row and the two far-field rows."""
        g, s = self.gam, q[:, 0]
        nx, ny = self.nj[0][0], self.nj[1][0]
        u, v = s[1] / s[0], s[2] / s[0]
        dn = 2 * (nx * u + ny * v)
        wall = torch.stack((s[0], s[0] * (u - dn * nx), s[0] * (v - dn * ny), s[3]))
        s, nx, ny = q[:, -1], self.nj[0][-1], self.nj[1][-1]
        rho, u, v = s[0], s[1] / s[0], s[2] / s[0]
        inout = nx * self.u + ny * self.v
        u2 = u * u + v * v
        a2 = g * (s[3] - 0.5 * u2 * rho) * (g - 1) / rho
        minf2 = self.u ** 2 + self.v ** 2
        un, ai = u * nx + v * ny, a2.clamp(min=0).sqrt()
        jp, jm = un + 2 * ai / (g - 1), inout - 2 / (g - 1)
        ag = torch.maximum(0.1 * ai, 0.25 * (jp - jm) * (g - 1))
        rg = (rho * (ag / ai).clamp(min=1e-6) ** 5).clamp(min=1e-6)
        d = 0.5 * (jp + jm) - un
        vx, vy = d * nx + u, d * ny + v
        sub = torch.stack((rg, vx * rg, vy * rg, (rg * ag * ag / g).clamp(min=1e-6) / (g - 1) + 0.5 * rg * (vx * vx + vy * vy)))
        if minf2 > 1:
            g1 = torch.stack((s[0], s[1], s[2], self.pin / (g - 1) + 0.5 * rho * u2))
        else:
            g1 = torch.where(u2 / a2 < 1, sub, s) if minf2 < 1 else s
        inflow = self.instate[:, None].expand_as(s)
        return wall, torch.where(inout < 0, inflow, g1), torch.where(inout < 0, inflow, 2 * g1 - s)

    def flux(self, L2, L, R, R2, n):
        if self.muscl:
            eps, dl, df, dr = 1e-6, L - L2, R - L, R2 - R
            den = df * df + eps
            rl, rr = (dl * df + eps) / den, (df * dr + eps) / den
            L, R = (L + 0.5 * (rl * rl + rl) / (rl * rl + 1) * df, R - 0.5 * (rr * rr + rr) / (rr * rr + 1) * df)
        g, nx, ny = self.gam, *n
        (rl, xl, yl, pl), (rr, xr, yr, pr) = L, R
        ul, ur, kl, kr = xl * nx + yl * ny, xr * nx + yr * ny, xl * xl + yl * yl, xr * xr + yr * yr
        hl, hr = pl / (0.4 * rl) + 0.5 * kl + pl / rl, pr / (0.4 * rr) + 0.5 * kr + pr / rr
        zero, one = torch.zeros_like(ul), torch.ones_like(ul)
        if self.scheme == "AUSM+-up":
            minf2 = (self.u ** 2 + self.v ** 2) / (g * self.pin / rl)
            a_s = (2 * 0.4 / (g + 1) * 0.5 * (hl + hr)).clamp(min=1e-6).sqrt()
            a = torch.minimum(a_s ** 2 / torch.maximum(ul, a_s), a_s ** 2 / torch.maximum(-ur, a_s))
            ml, mr = ul / a, ur / a
            mb = (ul * ul + ur * ur) / (2 * a * a)
            mo = torch.maximum(mb, minf2).clamp(max=1.0)
            fa = mo * (2 - mo)
            pml, pmr, mml, mmr = 0.25 * (ml + 1) ** 2, 0.25 * (mr + 1) ** 2, -0.25 * (ml - 1) ** 2, -0.25 * (mr - 1) ** 2
            sl, sr = ml.abs() >= 1, mr.abs() >= 1
            mi = torch.where(sl, ml.clamp(min=0), pml * (1 + 2 * mml)) + torch.where(sr, mr.clamp(max=0), mmr * (1 - 2 * pmr))
            al = 0.75 * (-4 + 5 * fa * fa)
            fl = torch.where(sl, torch.where(ml >= 0, one, zero), pml * ((2 - ml) + al * ml * mml))
            fr = torch.where(sr, torch.where(mr <= 0, one, zero), mmr * ((-2 - mr) - al * mr * pmr))
            P = fl * pl + fr * pr - 0.75 * fl * fr * (rl + rr) * fa * a * (ur - ul)
            m = a * mi * torch.where(mi > 0, rl, rr)
        else:
            a = 0.5 * ((g * pl.clamp(min=1e-10) / rl).sqrt() + (g * pr.clamp(min=1e-10) / rr).sqrt())
            ua = (0.5 * (kl + kr)).sqrt()
            ml, mr = ul / a, ur / a
            X = (1 - (ua / a).clamp(max=1.0)) ** 2
            bl, br = ml.clamp(-1, 1), mr.clamp(-1, 1)
            fp, fm = 0.25 * (bl + 1) ** 2 * (2 - bl), 0.25 * (br - 1) ** 2 * (2 + br)
            if self.scheme == "SLAU2":
                P = 0.5 * ((fp - fm) * (pl - pr) + (pl + pr) + ua * (fp + fm - 1) * (rl + rr) * a)
            else:
                P = 0.5 * ((fp - fm) * (pl - pr) + (1 + (1 - X) * (fp + fm - 1)) * (pl + pr))
            ub = (rl * ul.abs() + rr * ur.abs()) / (rl + rr)
            w = (-ml).clamp(0, 1) * mr.clamp(0, 1)
            m = 0.5 * ((rl * (ul + ub * (1 - w) + ul.abs() * w) + rr * (ur - ub * (1 - w) - ur.abs() * w)) * (1 - w)
                       - X / a * (pr - pl))
        left = m > 0
        return torch.stack((m, torch.where(left, xl, xr) * m + nx * P, torch.where(left, yl, yr) * m + ny * P,
                            torch.where(left, hl, hr) * m))

    def residual(self, q):
        wall, g1, g2 = self.ghosts(q)
        W = self.prim(torch.cat((wall[:, None], wall[:, None], q, g1[:, None], g2[:, None]), dim=1))
        fj = self.flux(W[:, :-3], W[:, 1:-2], W[:, 2:-1], W[:, 3:], self.nj) * self.lj
        W = W[:, 2:-2]
        fi = self.flux(W.roll(2, 2), W.roll(1, 2), W, W.roll(-1, 2), self.ni) * self.li
        return -(fi.roll(-1, 2) - fi + fj[:, 1:] - fj[:, :-1]) / self.A

    def max_wave(self):
        q = self.q
        k = (q[1] ** 2 + q[2] ** 2) / q[0] ** 2
        return float(((k.sqrt() + (self.gam * (q[3] - 0.5 * q[0] * k) * 0.4 / q[0]).sqrt()) * self.W).max())

    def step(self, n):
        dt = 0.5 / self.max_wave()
        for _ in range(n):
            q0 = self.q
            q1 = q0 + dt * self.residual(q0)
            q1 = 0.75 * q0 + 0.25 * (q1 + dt * self.residual(q1))
            self.q = (q0 + 2 * (q1 + dt * self.residual(q1))) / 3
        return dt

    def l2(self):
        return float(self.residual(self.q)[0].square().mean().sqrt())

    def wall_pressure(self):
        q = self.q[:, 0]
        return (q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) / q[0]) * 0.4

    def forces(self):
        p, x, y = self.wall_pressure(), self.g.x[0], self.g.y[0]
        fx, fy = float(-(p * (y.roll(-1) - y)).sum()), float((p * (x.roll(-1) - x)).sum())
        qi, sp = 0.5 * (self.u ** 2 + self.v ** 2), math.hypot(self.u, self.v)
        nx, ny = self.u / sp, self.v / sp
        return np.array([fx, fy, (-fx * ny + fy * nx) / qi, (fx * nx + fy * ny) / qi])

    def cp(self):
        return (self.wall_pressure() - self.pin) / (0.5 * (self.u ** 2 + self.v ** 2))

    def state(self):
        wall, g1, g2 = self.ghosts(self.q)
        return torch.cat((wall[:, None], self.q, g1[:, None], g2[:, None]), dim=1).permute(1, 2, 0).contiguous()


def exact_flow(d, rng, engine="fused"):
    g = Grid(d["M"], d["N"], d["naca"], far_radius(d), 1e-3, False)
    g.multicolor(d["sweeps"])
    if engine == "reference":
        g.rounded()
    f = Flow(g, d["mach"], d["aoa"], d["scheme"], d["muscl"])
    if rng is None:
        f.freestream()
    else:
        q = torch.from_numpy(disturbed_state(d["M"], d["N"], d["mach"], d["aoa"], rng)).cuda().double()
        f.q = q[1:-2].permute(2, 0, 1).contiguous()
    return f


def exact(case, seed):
    rng = np.random.RandomState(seed % (1 << 31))
    if case["kind"] == "frame":
        f = exact_flow(dict(case, **shape(rng, case)), rng, case["engine"])
        dt = f.step(case["n"])
        return dict(dt=dt, forces=f.forces(), state=f.state())
    if case["kind"] == "batch":
        dw, l2, states = [], [], []
        for d in batch_members(case, rng):
            f = exact_flow(d, rng)
            dw.append([f.step(case["n"]), f.max_wave()])
            l2.append(f.l2())
            states.append(f.state())
        return dict(dt_wave=np.array(dw), l2=np.array(l2), states=states)
    if case["kind"] == "serve":
        out = []
        for r in requests_of(case, rng):
            f = exact_flow(dict(r, muscl=1), None)
            for _ in range(case["steps"] // 100):
                f.step(100)
            out.append(dict(steps=None, stop=None, forces=f.forces(), Cp=f.cp()))
        return out
    d = dict(case, **shape(rng, case))
    g = Grid(d["M"], d["N"], d["naca"], 20.0, 1e-3, case["method"] == "jacobi")
    (g.jacobi if case["method"] == "jacobi" else g.multicolor)(case["sweeps"])
    return dict(done=None, vertices=g.vertices())
