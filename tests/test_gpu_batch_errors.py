"""Errors of batched simulations: a batch forms the next step's dt at the end
of a step, so a state whose CFL reduction fails (d <= 0 with eint > 0, which the
stage accepts) is met one step early.  As for a simulation alone, it is an error
of the step that starts from it: none for a simulation that ends on it, and none
before that step has run."""
import numpy as np
import pytest

from hormone_b200 import capi, config
from hormone_b200.batch import Batch, footprint
from hormone_b200.sim import Simulation

pytestmark = pytest.mark.gpu


def overrun(n, t_end):
    """Light gas behind dense gas at one speed and pressure, first order, one
    RK stage: a step longer than dx / v takes more mass out of the first dense
    cell than it holds, and leaves its internal energy as it was."""
    ov = dict(ie=n[0], je=n[1], ke=1, mag_on=False, gamma=1.4, courant=1.0, flux_limiter="flat", rktype=1, t_end=t_end,
              dt_out=t_end)
    for a in (1, 2, 3):
        for tag in ("is", "os", "iv", "ov"):
            ov[f"bc{a}{tag}"] = 3
    cfg = dict(config.resolve("riemann", overrides=ov), courant=8.0)  # past what the parameter file allows
    shape = (1, n[1], n[0])
    z = np.zeros(shape)
    d = z + 0.01
    d[:, :, n[0] // 2:] = 1.0
    return cfg, {"d": d, "p": z + 1.0, "v1": z + 10.0, "v2": z, "v3": z, "b1": z, "b2": z, "b3": z, "phi": z}


# few-item classes reduce in their last stage, the others (and the mixed form) in a kernel of their own
@pytest.mark.parametrize("n", [(64, 1), (18000, 1), (40, 9), (200, 150)])
@pytest.mark.parametrize("precision", [0, 1])
def test_bad_state_is_an_error_of_the_next_step(n, precision):
    last = overrun(n, 0.12 / n[0])  # ends on the bad state: 1.2 dx / v
    on = overrun(n, 1.0)
    b = Batch(footprint(last[0]) + footprint(on[0]) + (1 << 20), max_sims=3, precision=precision, rktype=1)
    sl, so = b.add(*last), b.add(*on)
    b.step(1)
    _, tn, done, err = b.poll()
    assert (tn[sl], done[sl], err[sl]) == (1, 1, 0)
    assert (tn[so], done[so], err[so]) == (1, 0, 0)
    got = b.download(sl)
    s = Simulation(*last, precision=precision)
    assert s.step()
    assert got["error"] == 0 and np.array_equal(got["u"], s.state()["u"]) and got["d"].min() <= 0.0
    s.close()
    b.step(9)
    _, tn, done, err = b.poll()
    assert (tn[sl], done[sl], err[sl]) == (1, 1, 0)
    assert err[so] == capi.HMN_ENEG_EINT
    b.close()
