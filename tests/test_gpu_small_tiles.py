"""The persistent small-grid loop's tiles (small_run_tile, hmn_small.cu): at
the sizes where the tile changes, and one cell around multiples of each tile,
whole steps must end on the same bits as the per-phase launches
(HMN_SMALL=0)."""
import numpy as np
import pytest

from hormone_b200 import config, grid as G, ic
from hormone_b200.sim import Simulation

import cases
from test_gpu_parity import run_pair

pytestmark = pytest.mark.gpu

# 1-D: 126 cells
# 2-D: 8x8 up to 296 tiles, then 16x16
# 3-D: 8x4x4 up to 148 tiles, then 8x8x8
SIZES = [(2, 1, 1), (29, 1, 1), (30, 1, 1), (31, 1, 1), (61, 1, 1), (4440, 1, 1), (4441, 1, 1), (37296, 1, 1),
         (37297, 1, 1), (7, 9, 1), (8, 8, 1), (9, 8, 1), (96, 96, 1), (96, 104, 1), (97, 97, 1), (256, 148, 1),
         (257, 149, 1), (7, 5, 3), (8, 4, 4), (9, 5, 5), (24, 24, 32), (25, 24, 40)]


def _case(n, mag):
    ov = dict(ie=n[0], je=n[1], ke=n[2], mag_on=mag, gamma=1.4, courant=0.6, t_end=1.0, dt_out=1.0)
    for a in (1, 2, 3):
        for tag in ("is", "os", "iv", "ov"):
            ov[f"bc{a}{tag}"] = (3, 0, 1)[a - 1]
    cfg = config.resolve("riemann", overrides=ov)
    rng = np.random.default_rng(sum(n))
    shape = (n[2], n[1], n[0])
    r = lambda lo, hi: rng.uniform(lo, hi, shape)  # noqa: E731
    z = np.zeros(shape)
    b = [r(-0.3, 0.3) if mag else z for _ in range(3)]
    if mag and n[1] == n[2] == 1:
        b[0] = z + 0.2  # the normal field of a 1-D grid is constant
    return cfg, {"d": r(0.8, 1.2), "p": r(0.8, 1.2), "v1": r(-0.3, 0.3), "v2": r(-0.3, 0.3), "v3": r(-0.3, 0.3),
                 "b1": b[0], "b2": b[1], "b3": b[2], "phi": z}


def _run(cfg, prims, steps):
    s = Simulation(cfg, prims)
    s.run_device(steps)
    out = s.state()["u"].copy(), s.time
    s.close()
    return out


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("mag", [False, True])
def test_tiles(monkeypatch, n, mag):
    cfg, prims = _case(n, mag)
    u, t = _run(cfg, prims, 3)
    monkeypatch.setenv("HMN_SMALL", "0")
    v, t0 = _run(cfg, prims, 3)
    assert t == t0 and np.array_equal(u, v)


@pytest.mark.parametrize("n", [(31, 1, 1), (127, 1, 1), (17, 16, 1), (40, 33, 1)])
def test_spherical_tiles(monkeypatch, n):
    cfg, prims = cases.spherical(n=n, mag=n[1] > 1)
    u, t = _run(cfg, prims, 3)
    monkeypatch.setenv("HMN_SMALL", "0")
    v, t0 = _run(cfg, prims, 3)
    assert t == t0 and np.array_equal(u, v)


# steps driven call by call take the small tiles of 1-D and 2-D grids too
# (launch_stage_few, hmn_kernels.cu): against the oracle
@pytest.mark.parametrize("n", [(30, 1, 1), (31, 1, 1), (4440, 1, 1), (4441, 1, 1), (8, 8, 1), (9, 7, 1), (96, 96, 1),
                               (97, 97, 1), (256, 149, 1)])
@pytest.mark.parametrize("mag", [False, True])
def test_host_driven_steps(n, mag):
    cfg, prims = _case(n, mag)
    run_pair(cfg, prims, 2)


@pytest.mark.parametrize("n", [(31, 1, 1), (17, 16, 1), (128, 80, 1)])
def test_host_driven_spherical_steps(n):
    cfg, prims = cases.spherical(n=n, mag=n[1] > 1)
    run_pair(cfg, prims, 2)
