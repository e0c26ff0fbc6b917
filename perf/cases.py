"""Performance cases: the work a host program has this framework do, through its public entry points.

A pass of a single-grid case is one run as a HORMONE host makes it: the conserved planes go to the device
(hmn_upload), a number of steps run (hmn_run, or the host's own loop over timestep, gravity, hydro_step and
phidamp), and the new planes come back into the host's arrays (hmn_download).  A batch case advances every
simulation of a running batch and collects all states; a serve case serves a whole stream of requests.

``exact`` computes the same passes with elementary torch operations in 64 bits.
"""
import ctypes
import math
import random

import numpy as np
import torch

from hormone_b200 import batch as batching
from hormone_b200 import capi, config, grid as gridmod, ic, serve as serving

FOREVER = 1e30  # end time: the number of steps bounds every run
PI = math.pi
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # Brio-Wu tube driven call by call, as the Fortran main loop drives the four procedures: launch latency
        dict(name="tube_1024_loop", kind="tube", nx=1024, ny=1, nz=1, precision=0, steps=4, loop="host"),
        # HORMONE's sedov_default test: a radial spherical grid, all steps on the device
        dict(name="sedov_500", kind="sedov", nx=500, ny=1, nz=1, precision=0, steps=64, loop="device"),
        # HORMONE's 2-D Orszag-Tang test
        dict(name="vortex_128sq", kind="vortex", nx=128, ny=128, nz=1, precision=0, steps=64, loop="device"),
        # Kelvin-Helmholtz with two passive scalars, odd sizes
        dict(name="shear_501x350_scalars", kind="shear", nx=501, ny=350, nz=1, precision=0, steps=32, loop="device"),
        # a ragged 3-D MHD box, the size of a quick resolution study
        dict(name="vortex_97x75x62", kind="vortex", nx=97, ny=75, nz=62, precision=0, steps=16, loop="device"),
        # the headline 3-D MHD box in FP64 ...
        dict(name="vortex_256", kind="vortex", nx=256, ny=256, nz=256, precision=0, steps=16, loop="device"),
        # ... and a 3-D MHD box in the mixed form
        dict(name="vortex_192_mixed", kind="vortex", nx=192, ny=192, nz=192, precision=1, steps=8, loop="device"),
        # many uneven 2-D boxes in one batch, both precisions
        dict(name="kh_batch", kind="batch", boxes=48, lo=128, hi=512, sizes=20261203, precision=0, steps=16),
        dict(name="kh_batch_mixed", kind="batch", boxes=48, lo=128, hi=512, sizes=20261203, precision=1, steps=16),
        # self-gravitating polytrope on a Cartesian box
        dict(name="polytrope_160", kind="polytrope", nx=160, ny=160, nz=160, precision=0, steps=8, loop="device"),
        # the same star on a spherical polar grid
        dict(name="star_128x64x128", kind="star", nx=128, ny=64, nz=128, precision=0, steps=8, loop="device"),
        # a served stream of small Riemann problems and blasts
        dict(name="serve_24", kind="serve", requests=24, cells=4096, sizes=20261203, precision=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "sedov", "vortex2", "vortex3", "vortex3", "shear", "blast", "batch", "polytrope", "star",
                       "serve"])
    c = dict(kind=kind, nx=1, ny=1, nz=1, precision=0, loop="device")
    if kind == "tube":
        c.update(nx=_log_int(rng, 100, 16384), precision=rng.randint(0, 1), steps=_log_int(rng, 4, 64),
                 loop=rng.choice(["host", "device"]))
    elif kind == "sedov":
        c.update(nx=_log_int(rng, 100, 4000), steps=_log_int(rng, 16, 128))
    elif kind == "vortex2":
        c.update(kind="vortex", nx=_log_int(rng, 60, 1200), ny=_log_int(rng, 60, 1200), precision=rng.randint(0, 1),
                 steps=_log_int(rng, 8, 64))
    elif kind == "vortex3":
        c.update(kind="vortex", nx=_log_int(rng, 24, 220), ny=_log_int(rng, 24, 220), nz=_log_int(rng, 24, 220),
                 precision=rng.randint(0, 1), steps=_log_int(rng, 8, 20), loop=rng.choice(["host", "device"]))
    elif kind == "shear":
        c.update(nx=_log_int(rng, 60, 1000), ny=_log_int(rng, 60, 1000), steps=_log_int(rng, 8, 40))
    elif kind == "blast":
        c.update(nx=_log_int(rng, 24, 200), ny=_log_int(rng, 24, 200), nz=_log_int(rng, 24, 200),
                 precision=rng.randint(0, 1), steps=_log_int(rng, 8, 16))
    elif kind == "batch":
        lo = _log_int(rng, 40, 160)
        c = dict(kind="batch", boxes=rng.randint(6, 48), lo=lo, hi=lo * 3, sizes=rng.randrange(1 << 20),
                 precision=rng.randint(0, 1), steps=_log_int(rng, 4, 16))
    elif kind == "polytrope":
        n = _log_int(rng, 32, 176)
        c.update(nx=n, ny=n, nz=n + rng.randint(-7, 7), steps=_log_int(rng, 4, 8))
    elif kind == "star":
        c.update(nx=_log_int(rng, 24, 140), ny=_log_int(rng, 16, 64), nz=_log_int(rng, 16, 128),
                 steps=_log_int(rng, 4, 8))
    else:
        c = dict(kind="serve", requests=rng.randint(8, 24), cells=_log_int(rng, 1000, 4096),
                 sizes=rng.randrange(1 << 20), precision=0)
    if c["precision"] and c["kind"] in ("vortex", "blast"):  # longer mixed passes differ by more than they say
        c["steps"] = min(c["steps"], 8)
    return c


# ---------------------------------------------------------------------------
# inputs

def _config(case):
    """The parameter set of a single-grid case."""
    k = case["kind"]
    ov = dict(ie=case["nx"], je=case["ny"], ke=case["nz"], t_end=FOREVER, dt_out=FOREVER)

    def faces(code):
        ov.update({"bc%d%s" % (a, t): code for a in (1, 2, 3) for t in ("is", "os", "iv", "ov")})

    if k == "tube":
        faces(3)
        ov.update(mag_on=True, gamma=2.0, courant=0.4, flux_limiter="minmod")
    elif k == "sedov":
        return config.resolve("sedov_default", overrides=dict(ov, dt_unit="s"))
    elif k == "vortex":
        ov.update(mag_on=True, gamma=1.6666666666666667, courant=0.9)
    elif k == "shear":
        return config.resolve("KHinstability", overrides=dict(ov, dt_unit="s"))
    elif k == "blast":
        faces(2)
        ov.update(gamma=1.4, courant=0.4, flux_limiter="minmod")
    elif k == "polytrope":
        faces(3)
        ov.update(gamma=2.0, gravswitch=3, G=1.0, courant=0.9, xi1s=-2.0, xi1e=2.0, xi2s=-2.0, xi2e=2.0, xi3s=-2.0,
                  xi3e=2.0)
    elif k == "star":
        ov.update(crdnt=2, gamma=2.0, gravswitch=3, gbtype=1, G=1.0, courant=0.9, xi1s=0.0, xi1e=2.0, bc1is=1, bc1iv=1,
                  bc1os=2, bc1ov=2)
    return config.resolve(k, overrides=ov)


def _inputs(case, seed):
    """(cfg, grid, u, spc, grvphi): the host's arrays before a single-grid run; u holds the conserved planes."""
    cfg = _config(case)
    grid = gridmod.make_grid(cfg)
    n = cfg["n"]
    shape = (n[2], n[1], n[0])
    rng = random.Random(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    f64 = dict(dtype=torch.float64, device=DEV)
    x, y, z = (torch.tensor(gridmod.centres(grid, a), **f64).reshape([-1 if 2 - a == d else 1 for d in range(3)])
               for a in range(3))
    zero = torch.zeros((), **f64)
    d = p = zero + 1.0
    v = [zero, zero, zero]
    b = [zero, zero, zero]
    spc = grvphi = None
    k = case["kind"]
    if k == "tube":  # Brio-Wu states, each moved by up to 10 %
        left = x < 0.5
        side = lambda l, r: torch.where(left, l * rng.uniform(0.9, 1.1), r * rng.uniform(0.9, 1.1))  # noqa: E731
        d, p = side(1.0, 0.125), side(1.0, 0.1)
        b = [zero + 0.75, side(1.0, -1.0), zero]
    elif k == "sedov":  # the blast energy in the first ten radial cells
        e = rng.uniform(0.5, 2.0)
        r0 = float(grid[0]["xi"][11])
        d = zero + rng.uniform(0.8, 1.2)
        p = torch.where(x < r0, 0.4 * e / (4.0 / 3.0 * PI * r0 ** 3), 1e-3 * e)
    elif k == "vortex":  # Orszag-Tang with seeded noise on the z components
        g = cfg["gamma"]
        d, p = zero + g * g / (4.0 * PI), zero + g / (4.0 * PI)
        noise = lambda: (torch.rand(shape, generator=gen, **f64) - 0.5) * 2e-3  # noqa: E731
        s4 = math.sqrt(4.0 * PI)
        v = [-torch.sin(2.0 * PI * y), torch.sin(2.0 * PI * x), noise()]
        b = [-torch.sin(2.0 * PI * y) / s4, torch.sin(4.0 * PI * x) / s4, noise()]
    elif k == "shear":  # exponential shear layers, each fluid marked by its own scalar
        ex = 0.5 * torch.exp(-(y.abs() - 0.25).abs() / 0.025)
        outer = y.abs() > 0.25
        d = torch.where(outer, 1.0 + ex, 2.0 - ex)
        p = zero + 2.5
        v = [torch.where(outer, 0.5 - ex, -0.5 + ex), 0.01 * rng.uniform(0.5, 2.0) * torch.sin(4.0 * PI * x), zero]
        mark = torch.where(outer, 1.0, 0.0) * torch.ones(shape, **f64)
        spc = torch.stack([mark, 1.0 - mark]).cpu().numpy()
    elif k == "blast":  # energy in a ball in cold gas at rest
        r2 = (x - 0.5) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2
        p = torch.where(r2 < 0.1 ** 2, 0.4 * rng.uniform(0.5, 2.0) / (4.0 / 3.0 * PI * 0.1 ** 3), 1e-5)
    else:  # the n=1 polytrope of unit radius in its own potential, the pressure off balance by up to 2 %
        r = x * torch.ones(shape, **f64) if k == "star" else torch.sqrt(x * x + y * y + z * z)
        poly = torch.where(r < 1.0, torch.sin(PI * r) / (PI * r), 0.0)
        d = poly.clamp(min=1e-6)
        p = 2.0 / PI * rng.uniform(0.98, 1.02) * poly * poly + 1e-6 * (4.0 / PI) / r.clamp(min=1.0)
        grvphi = torch.where(r < 1.0, -(4.0 / PI) * (1.0 + poly), -(4.0 / PI) / r).cpu().numpy()
    e = p / (cfg["gamma"] - 1.0) + 0.5 * (d * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2) + b[0] ** 2 + b[1] ** 2 + b[2] ** 2)
    planes = [d, d * v[0], d * v[1], d * v[2], e] + (b if cfg["mag_on"] else []) + ([zero] if cfg["glm"] else [])
    u = _host(len(planes), shape)
    for q, a in enumerate(planes):
        u[q].copy_(a.expand(shape))
    return cfg, grid, u.numpy(), spc, grvphi


def _host(nplanes, shape):
    """Host planes as a program that talks to a GPU keeps them: page-locked."""
    return torch.empty((nplanes,) + tuple(shape), dtype=torch.float64, pin_memory=DEV == "cuda")


def _boxes(case, seed):
    """(cfg, primitives) of each Kelvin-Helmholtz box of a batch: edges log-uniform in [lo, hi], given by the case;
    density ratio and field from the seed."""
    edges, rng = random.Random(case["sizes"]), random.Random(seed)
    out = []
    for _ in range(case["boxes"]):
        n = _log_int(edges, case["lo"], case["hi"])
        cfg = config.resolve("kh_batch", overrides=dict(ie=n, je=n, ke=1, mag_on=True, gamma=1.6666666666666667,
                                                        t_end=FOREVER, dt_out=FOREVER, xi1s=-0.5, xi1e=0.5, xi2s=-0.5,
                                                        xi2e=0.5))
        out.append((cfg, ic.kelvin_helmholtz(cfg, gridmod.make_grid(cfg), rng.uniform(1.0, 4.0), rng.uniform(0.0, 0.1))))
    return out


def _requests(case, seed):
    """A request stream whose sizes come from the case and whose states' strengths come from the seed."""
    rng = random.Random(seed)
    reqs = serving.make_requests(case["requests"], rate=50.0, seed=case["sizes"], max_cells=case["cells"])
    for r in reqs:
        f = rng.uniform(0.9, 1.1)
        r.prims = dict(r.prims, p=r.prims["p"] * f, d=r.prims["d"] * rng.uniform(0.9, 1.1))
    return reqs


# ---------------------------------------------------------------------------
# the passes

def prepare(case, seed):
    k = case["kind"]
    if k == "batch":
        boxes = _boxes(case, seed)
        pool = sum(batching.footprint(cfg) for cfg, _ in boxes) + (1 << 24)
        b = batching.Batch(pool, max_sims=len(boxes), precision=case["precision"])
        b.set_schedule(1, 2, 0)  # 16x16 tiles at the occupancy limit ...
        b.set_sweep(1, 2)        # ... taken from a shared counter: what the autotuner picks for 2-D boxes
        slots = [b.add(cfg, prims) for cfg, prims in boxes]
        outs = [_host(cfg["nvar"], (1, cfg["n"][1], cfg["n"][0])).numpy() for cfg, _ in boxes]
        return dict(case=case, batch=b, slots=slots, outs=outs)
    if k == "serve":
        reqs = _requests(case, seed)
        pool = sum(batching.footprint(r.cfg) for r in reqs) + (1 << 24)
        return dict(case=case, batch=batching.Batch(pool, max_sims=len(reqs), precision=case["precision"]),
                    requests=reqs)
    cfg, grid, u, spc, grvphi = _inputs(case, seed)
    state = dict(case=case, cfg=cfg, u=u, spc=spc, grvphi=grvphi, out=_host(*u.shape[:1], u.shape[1:]).numpy())
    if grvphi is not None:
        state["zeros"] = np.zeros_like(grvphi)
        state["gout"] = [_host(1, u.shape[1:]).numpy()[0] for _ in range(2)]
    state["ctx"] = capi.Context(cfg, grid, precision=case["precision"])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        for slot, out in zip(state["slots"], state["outs"]):
            _check(capi.lib().hmn_batch_download(b.h, slot, _ptr(out), None), "hmn_batch_download")
        return state["outs"]
    if case["kind"] == "serve":
        reqs = state["requests"]
        serving.serve(reqs, state["batch"], realtime=False, policy="priority")
        return {"request %02d" % r.rid: r.result["u"] for r in reqs if not r.error}
    ctx, cfg = state["ctx"], state["cfg"]
    ctx.upload(u=state["u"], grvphi=state["grvphi"], grvpsi=state.get("zeros"))
    if state["spc"] is not None:
        ctx.upload_scalars(state["spc"])
    if state["grvphi"] is not None:
        ctx.set_gravity_clock(0.0, 0.0)
    time = 0.0
    if case["loop"] == "host":  # the main loop of hormone.f90 without gravity
        for _ in range(case["steps"]):
            dt, _ch = ctx.timestep(time, FOREVER, FOREVER)
            ctx.hydro_step()
            if cfg["glm"]:
                ctx.phidamp()
            time += dt
    else:
        time, _steps = ctx.run(time, FOREVER, case["steps"])
    g = state.get("gout", [None, None])
    _check(capi.lib().hmn_download(ctx.h, _ptr(state["out"]), None, _ptr(g[0]), _ptr(g[1])), "hmn_download")
    got = {"u": state["out"], "time": time}
    if state["spc"] is not None:
        got["spc"] = ctx.download_scalars()
    if state["grvphi"] is not None:
        got.update(grvphi=g[0], grvpsi=g[1])
    return got


def _ptr(a):
    return None if a is None else a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _check(rc, where):
    if rc != 0:
        raise capi.HmnError(rc, where)


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what its results may differ by

def work(case):
    """Bytes: the state in and out of the device once a pass, and per RK stage the current state (and from the second
    stage on the step's first one) read and the new one written, since a state of any size but the smallest leaves
    the caches.  Flops: the scheme's operations, a quotient or square root counted once."""
    k = case["kind"]
    if k == "batch":
        edges = random.Random(case["sizes"])
        cells = sum(_log_int(edges, case["lo"], case["hi"]) ** 2 for _ in range(case["boxes"]))
        return _work(cells, 9, 2, case["steps"], cells * 9 * 8)
    if k == "serve":  # about one step per cell along the longest axis and speed, 3-D requests
        return _work(case["requests"] * case["cells"] // 4, 8, 2, 300, case["requests"] * case["cells"] * 2 * 18 * 8)
    cells = case["nx"] * case["ny"] * case["nz"]
    dim = sum(case[a] > 1 for a in ("nx", "ny", "nz"))
    nvar = {"tube": 8, "vortex": 9, "shear": 7}.get(k, 5)
    w = _work(cells, nvar, dim, case["steps"], 2 * cells * nvar * 8)
    if k in ("polytrope", "star"):  # about seven sub-cycles of two stages: phi, psi, rho read, phi, psi written
        w["bytes"] += case["steps"] * 14 * cells * 40
        w["flops"] += case["steps"] * 14 * cells * 28
    return w


def _work(cells, nvar, dim, steps, transfer):
    face, slope = (270, 170) if nvar >= 8 else (120, 100)
    return {"bytes": steps * cells * 8 * nvar * 8 + transfer, "flops": steps * 3 * cells * (dim * (face + slope) + 60)}


def tolerance(case):
    """The FP64 form promises the reference's results bit for bit.  The mixed form's FP32 fluxes move each step by about
    1e-8 of the state, and that decides the slope-zeroing tests differently in single cells: measured against ``exact``,
    a pass ends 1e-8 off on the tube, 2e-6 to 1.4e-5 on the smooth batched boxes, up to 5e-4 on the noisy vortex and the
    cold blast (largest single value 0.05)."""
    if case["precision"] == 0:
        return "exact"
    return {"tube": {"rel": 1e-6, "max": 1e-4}, "batch": {"rel": 6e-5, "max": 2e-3}}.get(
        case["kind"], {"rel": 2e-3, "max": 0.2})


# ---------------------------------------------------------------------------
# the same passes in plain 64-bit arithmetic

def exact(case, seed):
    k = case["kind"]
    if k == "serve":
        return None  # hundreds to thousands of steps of two dozen grids: minutes
    if k == "batch":
        few = 4
        outs = []
        for cfg, prims in _boxes(case, seed)[:few]:
            st = ic.to_state(cfg, prims)
            grid = _Plain(cfg, gridmod.make_grid(cfg), st["u"], prim=st["prim"])
            grid.run(case["steps"])
            outs.append(grid.planes())
        return outs + [None] * (case["boxes"] - len(outs))
    if case["nx"] * case["ny"] * case["nz"] * case["steps"] > 4e8:
        return None
    cfg, grid, u, spc, grvphi = _inputs(case, seed)
    s = _Plain(cfg, grid, u, spc=spc, grvphi=grvphi)
    s.run(case["steps"])
    got = {"u": s.planes(), "time": s.time}
    if spc is not None:
        got["spc"] = torch.stack(s.spc).cpu()
    if grvphi is not None:
        got.update(grvphi=s.gphi.cpu(), grvpsi=s.gpsi.cpu())
    return got


def _sign(s, x):
    return torch.copysign(torch.full_like(x, s), x)


def _min(a, b):
    return torch.where(a < b, a, b)


def _max(a, b):
    return torch.where(a > b, a, b)


def _rk(stage, kind):
    if kind == 3:
        return [(1.0, 1.0, 0.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0)][stage]
    return [(1.0, 1.0, 0.0), (0.5, 0.5, 0.5)][stage]


class _Plain:
    """One grid: MUSCL slopes, HLLD with GLM, SSP Runge-Kutta, CFL, hyperbolic gravity, passive scalars; Cartesian or
    spherical polar; boundary codes 0 to 3.  Arrays are (nz, ny, nx); dimension 2 - a runs along axis a."""

    def __init__(self, cfg, grid, u, prim=None, spc=None, grvphi=None):
        self.c, self.n, self.g = cfg, cfg["n"], grid
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64).to(DEV)  # noqa: E731
        self.u = [t(a) for a in u]
        self.mag, self.glm = cfg["mag_on"], cfg["glm"]
        self.gm1 = t(cfg["gamma"] - 1.0)  # a tensor: torch divides by a number through its reciprocal
        self.axes = [a for a in range(3) if cfg["solve"][a]]
        self.sph = cfg["crdnt"] == 2
        self.spc = [] if spc is None else [t(a) for a in spc]
        self.time, self.damp, self.ch = 0.0, 1.0, 0.0
        if prim is None:
            self.primitives()
        else:
            p = [t(a) for a in prim]
            self.d, self.v, self.e, self.b, self.phi = p[0], p[1:4], p[4], p[5:8], p[8]
            self.ei = self.eint(self.e, self.d, self.v, self.b)
        self.gphi = None
        if grvphi is not None:
            self.gphi = t(grvphi)
            self.gpsi = torch.zeros_like(self.gphi)
            self.gtime = self.cgrav_old = 0.0
            self.setup_gravity()

    def planes(self):
        return torch.stack(self.u).cpu()

    def along(self, a, key, lo, hi):
        """Axis a's array `key` at offsets lo .. hi - 1 (cell i at i + 2), shaped to broadcast."""
        s = [1, 1, 1]
        s[2 - a] = hi - lo
        return torch.as_tensor(self.g[a][key][lo:hi], dtype=torch.float64).to(DEV).reshape(s)

    def half(self, a, lo, hi):
        """x - (lower face) and (upper face) - x."""
        x = self.along(a, "x", lo, hi)
        return x - self.along(a, "xi", lo - 1, hi - 1), self.along(a, "xi", lo, hi) - x

    def eint(self, e, d, v, b):
        r = e - 0.5 * d * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
        return r - 0.5 * (b[0] * b[0] + b[1] * b[1] + b[2] * b[2]) if self.mag else r

    def primitives(self):
        u = self.u
        zero = torch.zeros_like(u[0])
        self.d, self.v, self.e = u[0], [u[q] / u[0] for q in (1, 2, 3)], u[4]
        self.b = u[5:8] if self.mag else [zero] * 3
        self.phi = u[8] if self.glm else zero
        self.ei = self.eint(self.e, self.d, self.v, self.b)

    # -- one axis ------------------------------------------------------------

    def ghosts(self, a, side):
        """The two cells beyond a face: (d, m1, m2, m3, e, b1, b2, b3, phi, eint, scalars...)."""
        n, bc = self.n[a], self.c["bc"][a][side]
        idx = {0: [n - 2, n - 1] if side == 0 else [0, 1], 1: [1, 0] if side == 0 else [n - 1, n - 2]}
        edge = [0, 0] if side == 0 else [n - 1, n - 1]
        pick = lambda t, code: t.index_select(2 - a, torch.tensor(idx.get(int(code), edge), device=DEV))  # noqa: E731
        d, p = pick(self.d, bc[0]), self.gm1 * pick(self.ei, bc[0])
        v, b = [pick(t, bc[1]) for t in self.v], [pick(t, bc[1]) for t in self.b]
        if bc[1] == 1:
            v[a], b[a] = -v[a], -b[a]
        elif bc[1] == 2 and side == 0:
            v[a] = _min(torch.zeros_like(v[a]), v[a]) if a == 0 else v[a] * (0.5 - _sign(0.5, v[a]))
        elif bc[1] == 2:
            v[a] = v[a] * (0.5 + _sign(0.5, v[a]))
        ei = p / self.gm1
        e = ei + 0.5 * (d * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + b[0] * b[0] + b[1] * b[1] + b[2] * b[2])
        return [d, d * v[0], d * v[1], d * v[2], e] + b + [pick(self.phi, bc[0]) * self.phifac, ei] + \
            [pick(s, bc[0]) for s in self.spc]

    def slope(self, a, um, u0, up):
        n = self.n[a]
        at = lambda key, o: self.along(a, key, 1 + o, n + 3 + o)  # noqa: E731  cells -1 .. n
        if self.c["limiter_code"] == 1:
            i0, i1 = at("idx", 0), at("idx", 1)
            x, y = 1.4 * (up - u0) * i1, 1.4 * (u0 - um) * i0
            z = (up - um) * i0 * i1 / (i0 + i1)
            s = _sign(1.0, x)
            m = _min(_min(x.abs(), s * y), s * z)
            return s * _max(torch.zeros_like(m), m)
        hl, hr = self.half(a, 1, n + 3)
        ga, gb = at("x", 1) - at("x", 0), at("x", 0) - at("x", -1)
        top, bot = (u0 - um) * ga / gb, up - u0
        s = _sign(1.0, bot)
        m = _min(_min(s * 0.5 * (bot + top), s * (ga / hr) * bot), s * (gb / hl) * top)
        return s * _max(torch.zeros_like(m), m) / ga

    def axis(self, a):
        """The fluxes through the n + 1 faces along axis a, conserved slots, then the scalars."""
        n, dim = self.n[a], 2 - a
        q = [self.d, self.d * self.v[0], self.d * self.v[1], self.d * self.v[2], self.e] + list(self.b) + \
            [self.phi * self.phifac, self.ei] + self.spc
        q = [torch.cat([l, t, h], dim) for l, t, h in zip(self.ghosts(a, 0), q, self.ghosts(a, 1))]
        cell = lambda t, lo: t.narrow(dim, lo, n + 2)  # noqa: E731
        vary = [0, 4, 1, 2, 3] + ([5, 6, 7] if self.mag else [])
        hl, hr = self.half(a, 1, n + 3)
        sl, lo, hi = {}, {}, {}
        for k in vary:
            um, u0, up = (cell(q[k], o) for o in (0, 1, 2))
            sl[k] = self.slope(a, um, u0, up)
            lo[k], hi[k] = u0 - hl * sl[k], u0 + hr * sl[k]
        inner = []
        for f in (lo, hi):
            ei = f[4] - 0.5 * (f[1] * f[1] + f[2] * f[2] + f[3] * f[3]) / f[0]
            inner.append(ei - 0.5 * (f[5] * f[5] + f[6] * f[6] + f[7] * f[7]) if self.mag else ei)
        em, e0, ep = (cell(q[9], o) for o in (0, 1, 2))
        off = (inner[0] >= _max(em, e0)) | (inner[0] <= _min(em, e0)) | (inner[1] >= _max(e0, ep)) | \
            (inner[1] <= _min(e0, ep))
        del lo, hi, inner
        zero = torch.zeros_like(em)
        sl = {k: torch.where(off, zero, s) for k, s in sl.items()}
        spsl = [self.slope(a, *(cell(t, o) for o in (0, 1, 2))) for t in q[10:]]
        dx1, dx2 = self.half(a, 1, n + 2)[1], self.half(a, 2, n + 3)[0]
        left = lambda t, s: t.narrow(dim, 1, n + 1) + dx1 * s.narrow(dim, 0, n + 1)  # noqa: E731
        right = lambda t, s: t.narrow(dim, 2, n + 1) - dx2 * s.narrow(dim, 1, n + 1)  # noqa: E731
        cn, c1, c2 = a, (a + 1) % 3, (a + 2) % 3
        st = []
        for f in (left, right):
            d, e = f(q[0], sl[0]), f(q[4], sl[4])
            v = [f(q[1 + c], sl[1 + c]) / d for c in (cn, c1, c2)]
            b = [f(q[5 + c], sl[5 + c]) for c in (cn, c1, c2)] if self.mag else [torch.zeros_like(d)] * 3
            ei = self.eint(e, d, v, b)
            p = self.gm1 * ei
            cs = torch.sqrt(self.c["gamma"] * p / d)
            pt = p + 0.5 * (b[0] * b[0] + b[1] * b[1] + b[2] * b[2])
            st.append((d, v, b, e, pt, self.fast(d, cs, *b), f(q[8], zero)))
        f = self.hlld(*st)
        out = [f[0], None, None, None, f[4], None, None, None, f[8]]
        for i, c in enumerate((cn, c1, c2)):
            out[1 + c], out[5 + c] = f[1 + i], f[5 + i]
        if self.spc:
            xl = [left(t, s) for t, s in zip(q[10:], spsl)]
            xr = [right(t, s) for t, s in zip(q[10:], spsl)]
            sg = _sign(0.5, f[0])
            fix = 1.0 / (sum(xl[1:], 0.0 + xl[0]) * (0.5 + sg) + sum(xr[1:], 0.0 + xr[0]) * (0.5 - sg))
            out += [fix * f[0] * (l * (0.5 + sg) + r * (0.5 - sg)) for l, r in zip(xl, xr)]
        return out

    @staticmethod
    def fast(d, cs, b1, b2, b3):
        asq, bb1 = cs * cs, b1 * b1 / d
        t = asq + (bb1 + b2 * b2 / d + b3 * b3 / d)
        return torch.sqrt(0.5 * (t + torch.sqrt(t * t - 4.0 * asq * bb1)))

    def hlld(self, left, right):
        ch = torch.tensor(self.ch, dtype=torch.float64, device=DEV)
        (dl, (v1l, v2l, v3l), (b1l, b2l, b3l), el, ptl, cfl, phil) = left
        (dr, (v1r, v2r, v3r), (b1r, b2r, b3r), er, ptr, cfr, phir) = right
        b1 = 0.5 * ((b1l + b1r) - (phir - phil) / ch)
        phi = 0.5 * ((phil + phir) - (b1r - b1l) * ch)
        zero = torch.zeros_like(dl)
        sl = _min(_min(v1r - cfr, v1l - cfl), zero)
        sr = _max(_max(v1r + cfr, v1l + cfl), zero)
        wl, wr = sl - v1l, sr - v1r
        den = wr * dr - wl * dl
        sm = (wr * dr * v1r - wl * dl * v1l - ptr + ptl) / den
        dla, dra = dl * wl / (sl - sm), dr * wr / (sr - sm)
        ql, qr = torch.sqrt(dla), torch.sqrt(dra)
        sla, sra = sm - b1.abs() / ql, sm + b1.abs() / qr
        pta = (wr * dr * ptl - wl * dl * ptr + dl * dr * wr * wl * (v1r - v1l)) / den
        star = []
        for d, w, s, v1, v2, v3, b2, b3, e, pt in ((dl, wl, sl, v1l, v2l, v3l, b2l, b3l, el, ptl),
                                                   (dr, wr, sr, v1r, v2r, v3r, b2r, b3r, er, ptr)):
            dd, num = d * w * (s - sm) - b1 * b1, d * w * w - b1 * b1
            v2a, v3a = v2 - b1 * b2 * (sm - v1) / dd, v3 - b1 * b3 * (sm - v1) / dd
            b2a, b3a = b2 * num / dd, b3 * num / dd
            ea = (w * e - pt * v1 + pta * sm +
                  b1 * ((v1 * b1 + v2 * b2 + v3 * b3) - (sm * b1 + v2a * b2a + v3a * b3a))) / (s - sm)
            star.append((v2a, v3a, b2a, b3a, ea))
        (v2la, v3la, b2la, b3la, ela), (v2ra, v3ra, b2ra, b3ra, era) = star
        s1, qs, qlr = _sign(1.0, b1), ql + qr, torch.sqrt(dla * dra)
        v2aa = (ql * v2la + qr * v2ra + (b2ra - b2la) * s1) / qs
        v3aa = (ql * v3la + qr * v3ra + (b3ra - b3la) * s1) / qs
        b2aa = (ql * b2ra + qr * b2la + qlr * (v2ra - v2la) * s1) / qs
        b3aa = (ql * b3ra + qr * b3la + qlr * (v3ra - v3la) * s1) / qs
        vb = v2aa * b2aa + v3aa * b3aa
        eraa = era + s1 * qr * ((v2ra * b2ra + v3ra * b3ra) - vb)
        elaa = ela - s1 * ql * ((v2la * b2la + v3la * b3la) - vb)
        wsl, wsr, wlr = 0.5 + _sign(0.5, sla), 0.5 + _sign(0.5, -sra), 0.5 - _sign(0.5, sla * sra)
        d = (0.5 + _sign(0.5, sm)) * dla + (0.5 - _sign(0.5, sm)) * dra
        v2, v3, b2, b3 = (wsl * l + wlr * m + wsr * r for l, m, r in
                          ((v2la, v2aa, v2ra), (v3la, v3aa, v3ra), (b2la, b2aa, b2ra), (b3la, b3aa, b3ra)))
        e = wsl * ela + (0.5 - _sign(0.5, sla * sm)) * elaa + (0.5 + _sign(0.5, -(sm * sra))) * eraa + \
            (0.5 - _sign(0.5, sra)) * era
        dv = d * sm
        return [dv, dv * sm + pta - b1 * b1, dv * v2 - b1 * b2, dv * v3 - b1 * b3,
                (e + pta) * sm - b1 * (sm * b1 + v2 * b2 + v3 * b3), phi, b2 * sm - b1 * v2, b3 * sm - b1 * v3,
                ch * ch * b1]

    # -- one step ------------------------------------------------------------

    def metric(self):
        """Spherical factors: dvol, the lower and upper face areas per axis, and per axis (cell weight, lower and
        upper face weight) of the divergence."""
        n0, n1, n2 = self.n
        fj, fk = 2.0 if n1 == 1 else 1.0, 4.0 if n2 == 1 else 1.0
        a, b = self.along(0, "xi", 2, n0 + 2), self.along(0, "xi", 1, n0 + 1)
        cd = self.along(1, "cosi", 1, n1 + 1) - self.along(1, "cosi", 2, n1 + 2)
        s0, s1 = self.along(1, "sini", 1, n1 + 1), self.along(1, "sini", 2, n1 + 2)
        dx2, dx3 = self.along(1, "dxi", 2, n1 + 2), self.along(2, "dxi", 2, n2 + 2)
        ar, three = a * a - b * b, torch.full_like(a, 3.0)
        dvol = (a * a * a - b * b * b) / three * cd * dx3 * fj * fk
        area = [(0.5 * (b * b) * cd * dx3 * fj * fk, 0.5 * (a * a) * cd * dx3 * fj * fk),
                (0.5 * s0 * ar * dx3 * fk, 0.5 * s1 * ar * dx3 * fk), (0.5 * ar * dx2 * fj, 0.5 * ar * dx2 * fj)]
        id2 = 1.0 / (-self.along(1, "cosi", 2, n1 + 2) + self.along(1, "cosi", 1, n1 + 1)) * self.along(0, "sx", 2, n0 + 2)
        div = [(self.along(0, "idetg", 2, n0 + 2), self.along(0, "detg", 1, n0 + 1), self.along(0, "detg", 2, n0 + 2)),
               (id2, s0, s1), (id2 * dx2 * self.along(2, "idxi", 2, n2 + 2) * (1.0 / fk), 1.0, 1.0)]
        return dvol, area, div

    def widths(self):
        return [self.along(a, "dxi", 2, self.n[a] + 2) for a in range(3)]

    def volumes(self):
        if self.sph:
            return self.metric()[:2]
        w = self.widths()
        s = [w[1] * w[2], w[0] * w[2], w[0] * w[1]]
        return w[0] * w[1] * w[2], [(x, x) for x in s]

    def timestep(self):
        c, d = self.c, self.d
        p = self.gm1 * self.ei
        cs = torch.sqrt(c["gamma"] * p / d)
        speed = [cs, cs, cs]
        if self.mag:  # the field components in the order (normal, then the other two ascending)
            speed = [self.fast(d, cs, *(self.b[k] for k in o)) for o in ((0, 1, 2), (1, 0, 2), (2, 0, 1))]
        cf = [s + v.abs() for s, v in zip(speed, self.v)]
        dvol, area = self.volumes()
        on = [1.0 if s else 0.0 for s in c["solve"]]
        t = [cf[a] * on[a] * (area[a][0] + area[a][1]) for a in range(3)]
        self.dt = c["courant"] * float((dvol / (t[0] + t[1] + t[2])).min())
        self.ch = float(_max(_max(cf[0], cf[1]), cf[2]).max())

    def source(self, acc):
        d, v, b = self.d, self.v, self.b
        n0, n1, _ = self.n
        frc = None if self.gphi is None else self.force()
        if not self.sph:
            if frc:
                for a in range(3):
                    acc[1 + a] = acc[1 + a] + frc[a]
                acc[4] = acc[4] + (frc[0] * v[0] + frc[1] * v[1] + frc[2] * v[2])
            return
        s1, sc = self.along(0, "sx", 2, n0 + 2), self.along(1, "scot", 2, n1 + 2)
        pt = self.gm1 * self.ei  # the spherical cases carry no field
        r = [(d * (v[1] * v[1] + v[2] * v[2]) + 2.0 * pt) * s1,
             (-(d * v[0] * v[1]) + (d * (v[2] * v[2]) + pt) * sc) * s1 if n1 > 1 else torch.zeros_like(d),
             (-(d * v[0] * v[2]) - d * v[1] * v[2] * sc) * s1]
        if frc:
            ss = self.along(1, "sisin", 2, n1 + 2)
            r = [r[0] + frc[0], r[1] + frc[1] * s1, r[2] + frc[2] * s1 * ss]
            acc[4] = acc[4] + (frc[0] * v[0] + frc[1] * v[1] * s1 + frc[2] * v[2] * s1 * ss)
        for a in range(3):
            acc[1 + a] = acc[1 + a] + r[a]

    def stage(self, s, org, sporg):
        faco, fact, facn = _rk(s, self.c["rktype"])
        self.phifac = self.damp if s == 0 else 1.0
        nv = len(self.u)
        acc = [torch.zeros_like(self.d) for _ in range(nv + len(self.spc))]
        div = self.metric()[2] if self.sph else None
        for a in self.axes:
            n, dim = self.n[a], 2 - a
            f = self.axis(a)
            f = f[:nv] + f[9:]
            for q in range(len(acc)):
                lo, hi = f[q].narrow(dim, 0, n), f[q].narrow(dim, 1, n)
                if self.sph:
                    acc[q] = acc[q] + div[a][0] * (div[a][1] * lo - div[a][2] * hi)
                else:
                    acc[q] = acc[q] + self.along(a, "idxi", 2, n + 2) * (lo - hi)
        self.source(acc)
        dtf = fact * self.dt
        din = self.d
        self.u = [faco * o + facn * c + dtf * x for o, c, x in zip(org, self.u, acc)]
        self.spc = [(faco * o + facn * x * din + dtf * g) / self.u[0] for o, x, g in zip(sporg, self.spc, acc[nv:])]
        self.primitives()

    def run(self, steps):
        for _ in range(steps):
            self.timestep()
            if self.gphi is not None:
                self.gravity()
            org, sporg = self.u, [x * self.u[0] for x in self.spc]
            for s in range(self.c["rktype"]):
                self.stage(s, org, sporg)
            self.damp = math.exp(-self.c["alpha9wave"] * self.c["courant"]) if self.glm else 1.0
            self.time = self.time + self.dt

    # -- self-gravity ----------------------------------------------------------

    def radius(self, off):
        """Distance from the origin of the cells at the given offsets (0: the cells, -1 / 1: one further) per axis."""
        x, y, z = (self.along(a, "x", 2 + o, self.n[a] + 2 + o) for a, o in enumerate(off))
        return torch.sqrt(x * x + y * y + z * z)

    def setup_gravity(self):
        n = self.n
        dvol, area = self.volumes()
        on = [1.0 if s else 0.0 for s in self.c["solve"]]
        t = [on[a] * (area[a][0] + area[a][1]) for a in range(3)]
        self.unit = float((dvol / (t[0] + t[1] + t[2])).min())
        if self.sph:
            cc, cx, cy, cz = (self.polar_weights(*o) for o in ((0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1)))
            self.c0, self.cn = cc[0], cc[4]
            self.cm, self.cp = [cx[1], cy[2], cz[3]], [cc[1], cc[2], cc[3]]
            return
        w = self.widths()
        i0 = [self.along(a, "idx", 2, n[a] + 2) + self.along(a, "idx", 3, n[a] + 3) for a in range(3)]
        self.c0 = -(i0[0] * w[1] * w[2] + i0[1] * w[0] * w[2] + i0[2] * w[0] * w[1]) + torch.zeros_like(self.d)
        ar = [w[1] * w[2], w[0] * w[2], w[0] * w[1]]
        self.cm = [(ar[a] / self.along(a, "dx", 2, n[a] + 2)).expand_as(self.d).clone() for a in range(3)]
        self.cp = [(ar[a] / self.along(a, "dx", 3, n[a] + 3)).expand_as(self.d).clone() for a in range(3)]
        self.cn = w[0] * w[1] * w[2]
        for a in range(3):  # phi ~ 1/r beyond each face, folded into the centre weight
            for c, o, at in ((self.cp[a], 1, n[a] - 1), (self.cm[a], -1, 0)):
                far = self.radius([o if b == a else 0 for b in range(3)])
                add = (c * self.radius([0, 0, 0]) / far).narrow(2 - a, at, 1)
                self.c0.narrow(2 - a, at, 1).add_(add)
                c.narrow(2 - a, at, 1).zero_()

    def polar_weights(self, di, dj, dk):
        """The spherical Laplacian's weights (centre, upper neighbour along each axis) and normalisation at cells
        displaced by (di, dj, dk)."""
        n0, n1, n2 = self.n
        r = lambda key, o=0: self.along(0, key, 2 + di + o, n0 + 2 + di + o)  # noqa: E731
        t = lambda key, o=0: self.along(1, key, 2 + dj + o, n1 + 2 + dj + o)  # noqa: E731
        f = lambda key, o=0: self.along(2, key, 2 + dk + o, n2 + 2 + dk + o)  # noqa: E731
        a, b, s, full = r("xi"), r("xi", -1), t("sinc"), torch.ones_like(self.d)
        rr = a * a / r("dx", 1) + b * b / r("dx")
        tt = t("sini") / t("dx", 1) + t("sini", -1) / t("dx")
        w1, w2, w3 = r("dxi"), t("dxi"), f("dxi")
        if n2 == 1:
            c0 = -(rr * s * w2 + tt * w1) * full
            c1, c2, c3 = a * a * s * w2 / r("dx", 1) * full, t("sini") * w1 / t("dx", 1) * full, 0.0 * full
            cn = r("x") * r("x") * s * w1 * w2
        else:
            c0 = -(rr * s * w2 * w3 + tt * w1 * w3 + (f("idx") + f("idx", 1)) * w1 * w2) * full
            c1, c2 = a * a * s * w2 * w3 / r("dx", 1) * full, t("sini") * w1 * w3 / t("dx", 1) * full
            c3 = w1 * w2 / f("dx", 1) * full
            cn = r("x") * r("x") * s * w1 * w2 * w3
        fold_t = n1 - 1 - dj  # the local index of the last theta cell
        if 0 <= fold_t < n1:
            c0[:, fold_t] += c2[:, fold_t]
            c2[:, fold_t] = 0.0
        last = n0 - 1 - di
        if 0 <= last < n0:
            x = self.g[0]["x"]
            c0[:, :, last] += c1[:, :, last] * float(x[n0 + 1]) / self.along(0, "x", n0 + 2, n0 + 3)[0]
            c1[:, :, last] = 0.0
        return c0, c1, c2, c3, cn

    def beyond(self, t, a, o):
        """t at the neighbour o = -1 / 1 along axis a, with the boundary's images of a potential."""
        dim, n = 2 - a, self.n[a]
        if n == 1:
            edge = t
        elif o < 0:
            edge = t.narrow(dim, 0, 1)
        else:
            edge = t.narrow(dim, n - 1, 1)
        if self.c["bc"][a][0][0] == 0:
            return torch.roll(t, -o, dim)
        if self.sph and a == 0 and o > 0:
            edge = edge * self.along(0, "x", n + 1, n + 2) / self.along(0, "x", n + 2, n + 3)
        elif not self.sph:
            at = 0 if o < 0 else n - 1
            far = self.radius([o if b == a else 0 for b in range(3)]).narrow(dim, at, 1)
            edge = edge * self.radius([0, 0, 0]).narrow(dim, at, 1) / far
        if n == 1:
            return edge
        return torch.cat([edge, t.narrow(dim, 0, n - 1)] if o < 0 else [t.narrow(dim, 1, n - 1), edge], dim)

    def force(self):
        out = []
        for a in range(3):
            n = self.n[a]
            pm, pp = self.beyond(self.gphi, a, -1), self.beyond(self.gphi, a, 1)
            dm, dp = self.along(a, "dx", 2, n + 2), self.along(a, "dx", 3, n + 3)
            im, ip = self.along(a, "idx", 2, n + 2), self.along(a, "idx", 3, n + 3)
            out.append(-((dm * ip * pp - dp * im * pm) / (dm + dp) + (dp - dm) * im * ip * self.gphi) * self.d)
        return out

    def gravity(self):
        c = self.c
        cg = c["HGfac"] * self.ch
        sub = min(self.dt, c["hgcfl"] * self.unit / cg)
        count = math.ceil((self.time + self.dt - self.gtime) / sub)
        if count < 1:
            return
        h = (self.time + self.dt - self.gtime) / float(count)
        src = 4.0 * PI * c["G"] * self.d
        for _ in range(count):
            damp = math.exp(-(1.0 - self.cgrav_old / cg + c["alphagrv"] * c["hgcfl"]))
            o1, o2 = self.gphi, self.gpsi
            for s in range(c["grktype"]):
                faco, fact, facn = _rk(s, c["grktype"])
                lap = self.c0 * self.gphi
                for a in range(3):  # weights beyond a closed face are zero
                    if self.sph and self.n[a] == 1:
                        continue
                    lap = lap + self.cm[a] * self.beyond(self.gphi, a, -1)
                    lap = lap + self.cp[a] * self.beyond(self.gphi, a, 1)
                fdc = fact * h * cg
                phi = faco * o1 + facn * self.gphi + fdc * self.gpsi
                psi = faco * o2 + facn * self.gpsi + fdc * (lap / self.cn - src)
                self.gphi, self.gpsi = phi, psi * damp if s == c["grktype"] - 1 else psi
            self.gtime, self.cgrav_old = self.gtime + h, cg
