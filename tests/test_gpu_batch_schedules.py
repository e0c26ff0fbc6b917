"""Schedules of FP64 classes that follow them, and where a class starts to.

A class of few items takes its own small tiles whatever the schedule, and the
boxes of test_gpu_batch.py are that small.  Here every class of a batch (1-D, 2-D
and 3-D, with and without a field) is past its line, with ragged edges on every
axis, and each simulation must end on the bits of the same run alone on every
tile, grid size and sweep."""
import numpy as np
import pytest

from hormone_b200 import autotune
from hormone_b200.batch import Batch, footprint

import cases
from test_gpu_batch import SCHEDULES
from test_gpu_batch_few import alone
from test_gpu_small_tiles import _case

pytestmark = pytest.mark.gpu
STEPS = 8


def per_step(b):
    """Launches of one step: rktype stages and a CFL reduction per class, the
    reduction in the last stage where the class has few items, and the clocks."""
    b.step(1)  # makes the work list and starts new simulations
    n = b.launches()
    b.step(1)
    return b.launches() - n


def open_blast(n):
    cfg, prims = cases.blast3d(n, bc=1, mag=False)
    return dict(cfg, t_end=1.0, dt_out=1.0), prims


@pytest.fixture(scope="module")
def sims():
    return [cases.kh2d(97), cases.kh2d(120, ratio=3.0), _case((150, 139, 1), False), cases.ot3d(29), open_blast(29),
            _case((17800, 1, 1), True), _case((17911, 1, 1), False)]


@pytest.fixture(scope="module")
def refs(sims):
    return [alone(c, p, STEPS) for c, p in sims]


@pytest.mark.parametrize("i", range(len(SCHEDULES)))
def test_schedules_give_each_simulation_its_own_bits(sims, refs, i):
    b = Batch(sum(footprint(c) for c, _ in sims) + (1 << 22), max_sims=8)
    slots = [b.add(c, p) for c, p in sims]
    autotune.apply(b, SCHEDULES[i])
    assert per_step(b) == 6 * 4 + 1  # two steps; no class on the small tiles
    autotune.apply(b, SCHEDULES[(i + 1) % len(SCHEDULES)])
    b.step(STEPS - 2)
    t, tn, _, err = b.poll()
    for s, (u, time) in zip(slots, refs):
        assert (tn[s], t[s], err[s]) == (STEPS, time, 0)
        assert np.array_equal(b.download(s)["u"], u), (i, s)
    b.close()


@pytest.mark.parametrize("n", [(25, 9, 9), (60, 50, 1), (300, 1, 1)])
def test_the_tuner_knows_where_a_class_follows_its_schedule(n):
    sim = _case(n, True)
    kind = autotune.grid_kind(sim[0])
    times = autotune.copies(kind, [sim], 0)
    for count, launches in ((times - 1, 4), (times, 5)):
        b = Batch(count * footprint(sim[0]) + (1 << 22), max_sims=count)
        for _ in range(count):
            b.add(*sim)
        assert per_step(b) == launches, (n, count)
        b.close()
