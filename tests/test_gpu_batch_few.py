"""Batch classes of few items (batch_few_tile, hmn_kernels.cu): small grids in a
batch run on smaller tiles whose last stage also reduces the next step's CFL
quantities.  Every simulation must end on the bits of the same run alone, on
both sides of the limits where the tile is chosen, with all three tile kinds
and both kinds of physics in one batch, across joining, holding and removing."""
import numpy as np
import pytest

from hormone_b200.batch import Batch, footprint
from hormone_b200.sim import Simulation

from test_gpu_small_tiles import _case

pytestmark = pytest.mark.gpu


def alone(cfg, prims, steps):
    s = Simulation(cfg, prims)
    s.run_device(steps)
    out = s.state()["u"].copy(), s.time
    s.close()
    return out


def check(b, slot, ref, where):
    u, t = ref
    assert b.poll()[0][slot] == t, where
    assert np.array_equal(b.download(slot)["u"], u), where


# items at the limits: 1-D 592 tiles of 30, 2-D 296 of 8x8, 3-D 148 of 8x4x4
@pytest.mark.parametrize("n", [(30, 1, 1), (31, 1, 1), (17760, 1, 1), (17761, 1, 1), (8, 8, 1), (9, 7, 1),
                               (128, 148, 1), (129, 148, 1), (8, 4, 4), (9, 5, 3), (32, 148, 4), (33, 148, 4)])
@pytest.mark.parametrize("mag", [False, True])
def test_one_simulation(n, mag):
    cfg, prims = _case(n, mag)
    b = Batch(footprint(cfg) + (1 << 20), max_sims=2)
    slot = b.add(cfg, prims)
    b.step(11)  # one graph of several steps and single ones
    check(b, slot, alone(cfg, prims, 11), (n, mag))
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("rktype", [1, 2, 3])
def test_mixed_classes_joining_holding_leaving(rktype, precision):
    sizes = [((40, 1, 1), True), ((33, 1, 1), False), ((16, 9, 1), True), ((10, 9, 1), False), ((9, 8, 5), True),
             ((8, 9, 6), False), ((64, 300, 1), True)]
    sims = []
    for n, mag in sizes:
        cfg, prims = _case(n, mag)
        sims.append((dict(cfg, rktype=rktype), prims))
    b = Batch(sum(footprint(c) for c, _ in sims) + (1 << 22), max_sims=8, precision=precision, rktype=rktype)

    def ref(i, steps):
        s = Simulation(sims[i][0], sims[i][1], precision=precision)
        for _ in range(steps):
            s.step()
        out = s.state()["u"].copy(), s.time
        s.close()
        return out

    slots = [b.add(*sims[i]) for i in range(4)]
    b.step(3)
    slots += [b.add(*sims[i]) for i in range(4, 7)]
    b.step(2)
    b.set_held([slots[0], slots[6]])
    b.step(9)
    b.set_held([])
    b.step(1)
    steps = [6, 15, 15, 15, 12, 12, 3]
    for i, slot in enumerate(slots):
        check(b, slot, ref(i, steps[i]), (rktype, precision, i))
    b.remove(slots[2])
    b.step(2)
    check(b, slots[1], ref(1, 17), "after a removal")
    b.close()
