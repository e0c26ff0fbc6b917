"""Both sides of every line where a small grid's tile changes, against the oracle,
bit for bit: the persistent loop (small_run_tile, hmn_small.cu: 126 cells; 8x8 up
to 296 tiles, then 16x16; 8x4x4 up to 148 tiles, then 8x8x8) and steps driven call
by call (launch_stage_few, hmn_kernels.cu: 30 cells up to 592 tiles, then 256; 8x8
up to 296 tiles with a field and 592 without, then 16x16), on Cartesian and
spherical grids.  Past the lines this is the only small-grid test of the larger
tiles' spherical kernels."""
import numpy as np
import pytest

from hormone_b200.sim import Simulation
from oracle.oracle import Oracle

import cases
from test_gpu_parity import run_pair
from test_gpu_small_tiles import _case

pytestmark = pytest.mark.gpu

LOOP = [(125, 1, 1), (126, 1, 1), (127, 1, 1), (253, 1, 1), (296, 64, 1), (297, 64, 1), (148, 4, 32), (32, 37, 16),
        (33, 37, 16)]
DRIVEN = [(17760, 1, 1), (17761, 1, 1), (296, 64, 1), (297, 64, 1), (296, 128, 1), (297, 128, 1)]
SPHERICAL = [(17760, 1, 1), (17761, 1, 1), (296, 64, 1), (297, 64, 1), (592, 64, 1), (593, 64, 1)]


def loop_against_oracle(cfg, prims, steps=3):
    o = Oracle(cfg)
    o.set_prims(prims)
    o.start()
    s = Simulation(cfg, prims)
    s.run_device(steps)
    for _ in range(steps):
        o.step()
    assert s.time == o.scalars()["time"]
    assert np.array_equal(s.state()["u"], o.u())
    s.close()


@pytest.mark.parametrize("mag", [False, True])
@pytest.mark.parametrize("n", LOOP)
def test_loop(n, mag):
    loop_against_oracle(*_case(n, mag))


@pytest.mark.parametrize("mag", [False, True])
@pytest.mark.parametrize("n", DRIVEN)
def test_driven(n, mag):
    run_pair(*_case(n, mag), 2)


@pytest.mark.parametrize("mag", [False, True])
@pytest.mark.parametrize("n", SPHERICAL)
def test_spherical(n, mag):
    if mag and n[1] == 1:
        pytest.skip("a radial grid carries no field here")
    cfg, prims = cases.spherical(n=n, mag=mag)
    run_pair(cfg, prims, 2)
    loop_against_oracle(cfg, prims, 2)
