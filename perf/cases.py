"""The measured workloads: what a user of this framework has it do.

Every case is one pass of a solver program through the public entry points:
advance some time steps, then read the results the program keeps (density,
velocity, and for immersed bodies the marker forces and the beams' state) into
its own page-locked host arrays. A pass continues from the state the last one
left, as a run does between two outputs.

Kinds (each also drawn at random sizes by ``draw``):

``cavity``    lid-driven cavity, no bodies: the plain lattice.
``channel``   velocity inlet, convective outlet, no-slip walls, no bodies.
``cylinder``  the same channel around one rigid circle of markers.
``filament``  the same channel around one clamped flexible filament.
``turek``     a rigid circle with a flexible tail behind it in a parabolic
              channel with a pressure outlet, one epsilon system for all
              markers: the arrangement of the reference's default case.
``ensemble``  many uneven channel cases stepped together as one batch.
``serve``     canopy solves submitted to the request server.

Lattice-only and rigid cases start from a seeded vortex field (a loaded
restart state), so every site holds a flow of its own; cases with flexible
bodies start as the framework starts them, with a seeded inlet velocity, and
have run past their start-up (200 steps, the ensemble's inlet ramp of 400)
before the pass, so that passes take alike many coupling iterations.
"""
import math

import numpy as np
import torch

from life_gb300.case import CONVECTIVE, PARABOLIC, PREC_NAMES, PRESSURE, VELOCITY, WALL, CaseParams, Circle, Filament
from life_gb300.configs import cavity, cylinder, filament, lattice_nu
from life_gb300.ensemble import canopy_case, ensemble_cases
from life_gb300.lib import Batch, Case, Server

CX = (0, 1, -1, 0, 0, 1, -1, 1, -1)
CY = (0, 0, 0, 1, -1, 1, -1, -1, 1)
W9 = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4
ELEM = {"f64": 8, "f32": 4, "f16": 2}


def listed():
    return [
        # the smallest call: one step of a lattice of the size a test or a first
        # try has, and its fields, as an interactive or coupled program asks for
        {"name": "channel_64x30_f64_step", "kind": "channel", "nx": 64, "ny": 30, "prec": "f64", "cm": True, "steps": 1},
        # the plain method at the size of the validation run (256 x 256, Re 1000)
        {"name": "cavity_256_f64", "kind": "cavity", "nx": 256, "ny": 256, "prec": "f64", "cm": False, "steps": 100},
        # a large run in the default storage form, central moments
        {"name": "cavity_1536_f64_cm", "kind": "cavity", "nx": 1536, "ny": 1536, "prec": "f64", "cm": True, "steps": 20},
        # the roofline workload: 4096 x 4096 in FP32
        {"name": "cavity_4096_f32", "kind": "cavity", "nx": 4096, "ny": 4096, "prec": "f32", "cm": False, "steps": 50},
        # half-precision storage, central moments, odd sizes
        {"name": "cavity_3001x2203_f16_cm", "kind": "cavity", "nx": 3001, "ny": 2203, "prec": "f16", "cm": True, "steps": 50},
        # an ordinary FP32 channel of odd size
        {"name": "channel_1501x703_f32", "kind": "channel", "nx": 1501, "ny": 703, "prec": "f32", "cm": False, "steps": 100},
        # the rigid-cylinder configuration in both of the forms it is run in,
        # 100 steps apart, as the force record of that run is
        {"name": "cylinder_f64", "kind": "cylinder", "nx": 1000, "ny": 400, "prec": "f64", "cm": True, "steps": 100,
         "d": 40},
        {"name": "cylinder_f32", "kind": "cylinder", "nx": 1000, "ny": 400, "prec": "f32", "cm": True, "steps": 100,
         "d": 40},
        # the flexible-filament configuration: FP32 lattice, FP64 beam
        {"name": "filament_f32", "kind": "filament", "nx": 1200, "ny": 400, "prec": "f32", "cm": False, "steps": 20,
         "length": 80},
        # the reference's default arrangement at its own lattice, plain form
        {"name": "turek_501x83_f64", "kind": "turek", "nx": 501, "ny": 83, "prec": "f64", "cm": False, "steps": 10,
         "d": 20, "length": 70},
        # the batched ensemble: 64 cases, rigid cylinders and filaments
        {"name": "ensemble_64_f32", "kind": "ensemble", "n": 64, "prec": "f32", "layout": 20260101, "steps": 20},
        # the request loop: canopy solves that arrive together
        {"name": "serve_6_f32", "kind": "serve", "n": 6, "prec": "f32", "layout": 7, "steps": 100},
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def steps(sites, prec, most):
        return max(1, min(most, int({"f64": 4.0e7, "f32": 6.0e8, "f16": 6.0e8}[prec] / sites)))

    kind = rng.choice(["cavity", "cavity", "channel", "channel", "cylinder", "cylinder", "filament", "turek", "ensemble",
                       "serve"])
    prec = rng.choice(["f64", "f32", "f32", "f16"])
    cm = rng.random() < 0.5
    if kind in ("cavity", "channel"):
        nx, ny = span(32, 4096), span(32, 4096)
        if prec == "f64":
            nx, ny = min(nx, 1900), min(ny, 1900)
        return {"kind": kind, "nx": nx, "ny": ny, "prec": prec, "cm": cm, "steps": steps(nx * ny, prec, span(1, 100))}
    if kind == "cylinder":
        d = span(12, 48)
        nx, ny = rng.randint(12 * d, 1100), rng.randint(5 * d, 500)
        return {"kind": kind, "nx": nx, "ny": ny, "prec": prec, "cm": cm, "steps": steps(nx * ny, prec, span(4, 100)),
                "d": d}
    if kind == "filament":
        length = rng.randint(20, 80)
        return {"kind": kind, "nx": rng.randint(8 * length, 1300), "ny": rng.randint(3 * length, 500),
                "prec": rng.choice(["f64", "f32"]), "cm": cm, "steps": rng.randint(1, 20), "length": length}
    if kind == "turek":
        d = rng.randint(12, 24)
        return {"kind": kind, "nx": rng.randint(22 * d, 700), "ny": rng.randint(4 * d, 140),
                "prec": rng.choice(["f64", "f32"]), "cm": cm, "steps": rng.randint(1, 10), "d": d,
                "length": rng.randint(2 * d, 3 * d)}
    if kind == "ensemble":
        return {"kind": kind, "n": span(3, 64), "prec": rng.choice(["f32", "f32", "f16"]),
                "layout": rng.randint(1, 10 ** 8), "steps": rng.randint(2, 20)}
    return {"kind": kind, "n": rng.randint(2, 6), "prec": rng.choice(["f64", "f32", "f32"]),
            "layout": rng.randint(1, 10 ** 8), "steps": rng.randint(10, 40)}


# ------------------------------------------------------------------ inputs --
def _speed(seed):
    """The seeded inlet or lid velocity, near the configurations' 0.04-0.05."""
    return float(np.random.Generator(np.random.PCG64(seed)).uniform(0.038, 0.046))


def _setup(case, seed):
    """(params, bodies) of a single-case kind."""
    kind, nx, ny = case["kind"], case["nx"], case["ny"]
    prec = PREC_NAMES[case["prec"]]
    u = _speed(seed)
    if kind == "cavity":
        p = cavity(precision=prec, cm=case["cm"])
        return p.replace(Nx=nx, Ny=ny, height_p=float(ny - 1), uxInlet_p=2.0 * u), []
    if kind in ("channel", "cylinder"):
        p, bodies = cylinder(precision=prec)
        p = p.replace(Nx=nx, Ny=ny, height_p=float(ny - 1), central_moments=case["cm"], uxInlet_p=u)
        if kind == "channel":
            return p, []
        d = case["d"]
        return p, [Circle(x=round(nx / 5.0, 2), y=round(ny / 2.0 + 0.3, 2), radius=d / 2.0)]
    if kind == "filament":
        L = case["length"]
        p, bodies = filament(precision=prec)
        p = p.replace(Nx=nx, Ny=ny, height_p=float(ny - 1), central_moments=case["cm"], uxInlet_p=u, ref_L=float(L),
                      initial_deflect=None, ux0_p=u)
        stiff = 0.2 * u * u * L ** 3 * 12.0
        return p, [Filament(x=round(nx / 4.0, 2), y=round(ny / 2.0, 2), length=float(L), height=1.0,
                            angle_deg=3.0, flexible=True, n_elements=L, clamped=True, rho=0.5 * L, E=stiff)]
    # turek: a stiff tail of the reference's proportions behind the circle
    d, L = case["d"], case["length"]
    omega = 1.0 / 0.6
    x, y = 2.0 * d + 0.5, round(ny / 2.0 - 0.4, 2)
    p = CaseParams(Nx=nx, Ny=ny, height_p=float(ny - 1), rho_p=1.0, nu_p=lattice_nu(omega), omega=omega,
                   wall_left=VELOCITY, wall_right=PRESSURE, wall_bottom=WALL, wall_top=WALL, profile=PARABOLIC,
                   uxInlet_p=u, inlet_ramp=400.0, uni_epsilon=True, central_moments=case["cm"], precision=prec,
                   ref_L=float(d), subTol=2e-9)
    return p, [Circle(x=x, y=y, radius=d / 2.0, ID=0),
               Filament(x=x + d / 2.0, y=y, length=float(L), height=4.0, angle_deg=0.0, flexible=True, n_elements=None,
                        clamped=True, rho=10.0, E=40.0, ID=1)]


def _flow(p, seed, u0):
    """A seeded flow in the reference layout (torch, FP64): density near 1, a
    divergence-free vortex field around the mean (u0, 0), and populations at
    equilibrium plus a small non-equilibrium part."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    x = torch.arange(p.Nx, dtype=torch.float64, device=dev)[:, None] * (2.0 * math.pi / p.Nx)
    y = torch.arange(p.Ny, dtype=torch.float64, device=dev)[None, :] * (2.0 * math.pi / p.Ny)
    ux = torch.full((p.Nx, p.Ny), u0, dtype=torch.float64, device=dev)
    uy = torch.zeros((p.Nx, p.Ny), dtype=torch.float64, device=dev)
    rho = torch.ones((p.Nx, p.Ny), dtype=torch.float64, device=dev)
    for _ in range(4):
        kx, ky = int(rng.integers(1, 6)), int(rng.integers(1, 6))
        a, b = rng.uniform(0.0, 2.0 * math.pi, 2)
        amp = rng.uniform(0.002, 0.006)
        # stream function amp / hypot * sin(kx x + a) sin(ky y + b), per lattice unit
        gx, gy = kx / p.Nx, ky / p.Ny
        s = amp / math.hypot(gx, gy)
        ux += s * gy * torch.sin(kx * x + a) * torch.cos(ky * y + b)
        uy -= s * gx * torch.cos(kx * x + a) * torch.sin(ky * y + b)
        rho += 2e-4 * torch.sin(kx * x + b) * torch.sin(ky * y + a)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    f = torch.empty((p.Nx, p.Ny, 9), dtype=torch.float64, device=dev)
    usq = ux * ux + uy * uy
    for v in range(9):
        cu = CX[v] * ux + CY[v] * uy
        f[:, :, v] = W9[v] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq)
        f[:, :, v] += (W9[v] * 1e-5) * torch.randn((p.Nx, p.Ny), dtype=torch.float64, device=dev, generator=gen)
    n = p.Nx * p.Ny
    rho = f.sum(dim=2)
    ux = (f[:, :, 1] - f[:, :, 2] + f[:, :, 5] - f[:, :, 6] + f[:, :, 7] - f[:, :, 8]) / rho
    uy = (f[:, :, 3] - f[:, :, 4] + f[:, :, 5] - f[:, :, 6] - f[:, :, 7] + f[:, :, 8]) / rho
    return rho.reshape(n), torch.stack([ux, uy], dim=2).reshape(n, 2), f.reshape(n, 9)


def _mean_flow(case, p):
    return 0.0 if case["kind"] == "cavity" else p.uxInlet_p


def _many(case, seed):
    """The (params, bodies) list of an ensemble or a serve case: the layout is
    the case's, the inlet velocities are the seed's."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if case["kind"] == "ensemble":
        cases = ensemble_cases(case["n"], seed=case["layout"], precision=PREC_NAMES[case["prec"]])
    else:
        lay = np.random.Generator(np.random.PCG64(case["layout"]))
        cases = [canopy_case(lay, precision=PREC_NAMES[case["prec"]])[:2] for _ in range(case["n"])]
    return [(p.replace(uxInlet_p=p.uxInlet_p * float(rng.uniform(0.96, 1.0)), ux0_p=0.0), b) for p, b in cases]


def _host(shape):
    """A host array of the program's own, page-locked when there is a GPU."""
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _buffers(params):
    """One density and one velocity array for all of a program's cases, and
    each case's part of them."""
    sizes = [p.Nx * p.Ny for p in params]
    rho, u = _host((sum(sizes),)), _host((sum(sizes), 2))
    ends = np.cumsum(sizes)
    return {"rho": rho, "u": u}, [{"rho": rho[e - n:e], "u": u[e - n:e]} for n, e in zip(sizes, ends)]


def prepare(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        batch = Batch(_many(case, seed))
        batch.step(400)
        views = [batch.case(k) for k in range(len(batch))]
        whole, parts = _buffers([v.params for v in views])
        return {"batch": batch, "views": views, "whole": whole, "parts": parts, "steps": steps}
    if kind == "serve":
        cases = _many(case, seed)
        whole, parts = _buffers([p for p, _ in cases])
        return {"server": Server(160 << 30), "cases": cases, "whole": whole, "parts": parts, "steps": steps}
    p, bodies = _setup(case, seed)
    c = Case(p, bodies)
    if kind in ("cavity", "channel", "cylinder"):
        c.set_fields(0, *[a.cpu().numpy() for a in _flow(p, seed, _mean_flow(case, p))])
    else:
        c.step(200)
    whole, parts = _buffers([p])
    return {"case": c, "whole": whole, "parts": parts, "steps": steps}


# --------------------------------------------------------------------- run --
def run(state):
    out = dict(state["whole"])
    if "batch" in state:
        state["batch"].step(state["steps"])
        for view, part in zip(state["views"], state["parts"]):
            view.fields(("rho", "u"), out=part)
        return out
    if "server" in state:
        s = state["server"]
        ids = [s.submit(p, b, state["steps"]) for p, b in state["cases"]]
        markers = []
        for rid, part in zip(ids, state["parts"]):
            s.wait(rid)
            with s.take(rid) as c:
                c.fields(("rho", "u"), out=part)
                markers.append(c.markers())
        for k in ("pos", "force"):
            out[k] = np.concatenate([m[k] for m in markers])
        return out
    c = state["case"]
    c.step(state["steps"])
    c.fields(("rho", "u"), out=state["parts"][0])
    if c.n_markers:
        out["force"] = c.markers()["force"]
    for k in range(c.n_flex):
        beam = c.fem(k)
        out["U%d" % k], out["Udot%d" % k] = beam["U"], beam["Udot"]
    return out


# -------------------------------------------------------------------- work --
def work(case):
    """Per step each population read once and written once, and the collision's
    arithmetic; once per pass the outputs."""
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        ps = [(p.Nx * p.Ny, p.central_moments) for p, _ in _many(case, 1)]
    else:
        ps = [(case["nx"] * case["ny"], case["cm"])]
    sites = sum(n for n, _ in ps)
    flops = sum(n * (250 if cm else 115) for n, cm in ps)
    return {"bytes": float(case["steps"] * sites * 18 * ELEM[case["prec"]] + 24 * sites),
            "flops": float(case["steps"] * flops)}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """Lattice-only and rigid-body passes in 64-bit torch. Flexible bodies have
    none: the beam's Newton and relaxation loops in plain torch take minutes."""
    if case["kind"] not in ("cavity", "channel", "cylinder"):
        return None
    p, bodies = _setup(case, seed)
    rho, u, f = _flow(p, seed, _mean_flow(case, p))
    shape = (p.Nx, p.Ny)
    s = _Plain(p, bodies, rho.reshape(shape), u.reshape(*shape, 2), f.reshape(*shape, 9).permute(2, 0, 1).contiguous())
    for _ in range(case["steps"]):
        s.step()
    n = p.Nx * p.Ny
    out = {"rho": s.rho.reshape(n), "u": torch.stack([s.ux, s.uy], dim=2).reshape(n, 2)}
    if bodies:
        out["force"] = s.marker_force
    return out


def _delta(r):
    a = r.abs()
    inner = (1.0 + torch.sqrt((1.0 - 3.0 * a * a).clamp_min(0.0))) / 3.0
    outer = (5.0 - 3.0 * a - torch.sqrt((1.0 - 3.0 * (1.0 - a) ** 2).clamp_min(0.0))) / 6.0
    return torch.where(a > 1.5, torch.zeros_like(a), torch.where(a > 0.5, outer, inner))


class _Plain:
    """The D2Q9 lattice step (BGK or central moments, no-slip and velocity
    walls with the regularised condition, convective right outlet) and the
    implicit immersed boundary of one rigid circle, in torch FP64 over arrays
    [9][Nx][Ny]."""

    def __init__(self, p, bodies, rho, u, f):
        self.p, self.f, self.rho = p, f, rho
        self.ux, self.uy = u[:, :, 0].clone(), u[:, :, 1].clone()
        self.fx = torch.zeros_like(rho)
        self.fy = torch.zeros_like(rho)
        self.dev = rho.device
        self.circle = bodies[0] if bodies else None
        if self.circle:
            self._markers(self.circle)

    def _eq(self, rho, ux, uy):
        if self.p.central_moments:
            def axis(c, w):
                return 9.0 * c * c * w * w + 6.0 * c * w - 3.0 * w * w + 2.0
            return torch.stack([0.25 * rho * W9[v] * axis(CX[v], ux) * axis(CY[v], uy) for v in range(9)])
        out = []
        for v in range(9):
            cu = CX[v] * ux + CY[v] * uy
            out.append(W9[v] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy)))
        return torch.stack(out)

    def _collide(self):
        om, f, rho, ux, uy, fx, fy = self.p.omega, self.f, self.rho, self.ux, self.uy, self.fx, self.fy
        if not self.p.central_moments:
            eq = self._eq(rho, ux, uy)
            out = []
            for v in range(9):
                cu = CX[v] * ux + CY[v] * uy
                g = 3.0 * W9[v] * (fx * (CX[v] - ux + 3.0 * CX[v] * cu) + fy * (CY[v] - uy + 3.0 * CY[v] * cu))
                out.append(f[v] + om * (eq[v] - f[v]) + (1.0 - 0.5 * om) * g)
            return torch.stack(out)
        # relax the central moments, then back through the raw moments
        k4 = sum(f[v] * ((CX[v] - ux) ** 2 - (CY[v] - uy) ** 2) for v in range(9)) * (1.0 - om)
        k5 = sum(f[v] * (CX[v] - ux) * (CY[v] - uy) for v in range(9)) * (1.0 - om)
        k3 = 2.0 * rho / 3.0
        kap = {(0, 0): rho, (1, 0): 0.5 * fx, (0, 1): 0.5 * fy, (2, 0): 0.5 * (k3 + k4), (0, 2): 0.5 * (k3 - k4),
               (1, 1): k5, (2, 1): fy / 6.0, (1, 2): fx / 6.0, (2, 2): rho / 9.0}
        raw = {}
        for a in range(3):
            for b in range(3):
                raw[a, b] = sum(math.comb(a, i) * math.comb(b, j) * ux ** (a - i) * uy ** (b - j) * kap[i, j]
                                for i in range(a + 1) for j in range(b + 1))

        def axis(c):  # the 1-D inverse: coefficients of the moments 0, 1, 2
            return (1.0, 0.0, -1.0) if c == 0 else (0.0, 0.5 * c, 0.5)
        return torch.stack([sum(axis(CX[v])[a] * axis(CY[v])[b] * raw[a, b] for a in range(3) for b in range(3)
                                if axis(CX[v])[a] != 0.0 and axis(CY[v])[b] != 0.0) for v in range(9)])

    def _moments(self, f):
        rho = f.sum(dim=0)
        mx = (f[1] - f[2]) + (f[5] - f[6]) + (f[7] - f[8])
        my = (f[3] - f[4]) + (f[5] - f[6]) + (f[8] - f[7])
        return rho, mx, my

    def _wall(self, f, nx, ny, un, rho=None):
        """The regularised condition on sites f [9][m] with inward normal
        (nx, ny) and velocity un; at a corner the density is given."""
        corner = nx != 0 and ny != 0
        if not corner:
            cn = [CX[v] * nx + CY[v] * ny for v in range(9)]
            plus = sum(f[v] for v in range(9) if cn[v] == -1)
            zero = sum(f[v] for v in range(9) if cn[v] == 0)
            rho = (2.0 * plus + zero) / (1.0 - (nx * un[0] + ny * un[1]))
        eq = self._eq(rho, un[0], un[1])
        opp = (0, 2, 1, 4, 3, 6, 5, 8, 7)
        g = [f[v] for v in range(9)]
        for v in range(9):  # in order: an opposite population may already be set
            if corner and (CX[v] == nx or CY[v] == ny):
                g[v] = eq[v] if nx * CX[v] + ny * CY[v] == 0 else eq[v] + g[opp[v]] - eq[opp[v]]
            elif not corner and cn[v] == 1:
                g[v] = eq[v] + g[opp[v]] - eq[opp[v]]
        neq = [g[v] - eq[v] for v in range(9)]
        sxx = sum(CX[v] ** 2 * neq[v] for v in range(9))
        syy = sum(CY[v] ** 2 * neq[v] for v in range(9))
        sxy = sum(CX[v] * CY[v] * neq[v] for v in range(9))
        return torch.stack([eq[v] + 4.5 * W9[v] * ((CX[v] ** 2 - 1 / 3) * sxx + (CY[v] ** 2 - 1 / 3) * syy
                                                   + 2.0 * CX[v] * CY[v] * sxy) for v in range(9)])

    def step(self):
        p = self.p
        nx, ny = p.Nx, p.Ny
        fs = self._collide()
        last, ux0, uy0 = self.f, self.ux, self.uy
        f = torch.stack([torch.roll(fs[v], (CX[v], CY[v]), (0, 1)) for v in range(9)])
        zero = torch.zeros(1, dtype=torch.float64, device=self.dev)
        r_in, mx, my = self._moments(f)  # of the fluid sites
        new = f.clone()
        # left and right columns (the y walls own the corners)
        if p.wall_left == VELOCITY:
            u_l = torch.full((ny - 2,), p.uxInlet_p, dtype=torch.float64, device=self.dev)
        else:
            u_l = torch.zeros(ny - 2, dtype=torch.float64, device=self.dev)
        new[:, 0, 1:-1] = self._wall(f[:, 0, 1:-1], 1, 0, (u_l, torch.zeros_like(u_l)))
        if p.wall_right == CONVECTIVE:
            out = ux0[nx - 1, :].mean()
            d = [(-0.5 * out) * (3.0 * a[nx - 1] - 4.0 * a[nx - 2] + a[nx - 3]) for a in (ux0, uy0)]
            for v in (2, 6, 8):
                c = last[v, nx - 1, :] + 3.0 * W9[v] * (d[0] * CX[v] + d[1] * CY[v])
                new[v, nx - 1, 1:-1] = c[1:-1]
        else:
            z = torch.zeros(ny - 2, dtype=torch.float64, device=self.dev)
            new[:, nx - 1, 1:-1] = self._wall(f[:, nx - 1, 1:-1], -1, 0, (z, z))
        # bottom and top rows and their corners
        for j, n, kind in ((0, 1, p.wall_bottom), (ny - 1, -1, p.wall_top)):
            lid = p.uxInlet_p if kind == VELOCITY else 0.0
            uw = torch.full((nx - 2,), lid, dtype=torch.float64, device=self.dev)
            new[:, 1:-1, j] = self._wall(f[:, 1:-1, j], 0, n, (uw, torch.zeros_like(uw)))
            for i, m in ((0, 1), (nx - 1, -1)):
                rc = 2.0 * r_in[i + m, j + n] - r_in[i + 2 * m, j + 2 * n]
                new[:, i, j] = self._wall(f[:, i, j, None], m, n, (zero + lid, zero), rc.reshape(1))[:, 0]
        self.f = new
        self.rho, mx, my = self._moments(new)
        self.ux, self.uy = mx / self.rho, my / self.rho
        if self.circle:
            self._bodies(mx, my)

    def _markers(self, c):
        n = int(math.floor(2.0 * math.pi * c.radius))
        k = torch.arange(n, dtype=torch.float64, device=self.dev) * (2.0 * math.pi / n)
        x, y = c.x + c.radius * torch.cos(k), c.y + c.radius * torch.sin(k)
        off = torch.arange(-2, 3, device=self.dev)
        i = torch.round(x).long()[:, None] + off
        j = torch.round(y).long()[:, None] + off
        dx, dy = _delta(x[:, None] - i), _delta(y[:, None] - j)
        self.wgt = dx[:, :, None] * dy[:, None, :]  # [n][5][5], zero outside the support
        self.si = i[:, :, None].expand(-1, 5, 5)
        self.sj = j[:, None, :].expand(-1, 5, 5)
        dist = torch.hypot(x[:, None] - x[None, :], y[:, None] - y[None, :])
        dist.fill_diagonal_(10.0)
        self.ds = dist.min(dim=1).values.clamp_max(10.0)
        px = _delta(x[None, None, :] - i[:, :, None])  # [n][5][markers]
        py = _delta(y[None, None, :] - j[:, :, None])
        a = torch.einsum("kab,kam,kbm->km", self.wgt, px, py) * self.ds[None, :]
        self.eps = torch.linalg.solve(a, torch.ones(n, dtype=torch.float64, device=self.dev))

    def _bodies(self, mx, my):
        at = (self.si, self.sj)
        force = []
        for q, m in enumerate((self.ux, self.uy)):
            force.append(-2.0 * ((self.rho * m)[at] * self.wgt).sum(dim=(1, 2)))
        self.marker_force = torch.stack(force, dim=1)
        spread = []
        for q in range(2):
            g = torch.zeros_like(self.rho)
            g.index_put_(at, (force[q] * self.eps * self.ds)[:, None, None] * self.wgt, accumulate=True)
            spread.append(g)
        self.fx, self.fy = spread
        self.ux, self.uy = (mx + 0.5 * self.fx) / self.rho, (my + 0.5 * self.fy) / self.rho
