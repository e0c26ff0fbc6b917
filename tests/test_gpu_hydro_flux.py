"""The flux of grids without a magnetic field against the CPU oracle, bit for
bit.  The stages form it from the two star states of the contact wave
(hllc, hormone_b200/csrc/hmn_math.cuh) where the oracle runs the full
five-wave solver with zero fields, and leave operands far from 1 to the full
solver: the cases put the state's scales inside, at and beyond those limits,
and the flow at rest, sub- and supersonic either way, in 1-D to 3-D."""
import numpy as np
import pytest

from hormone_b200 import config

from test_gpu_parity import run_pair

pytestmark = pytest.mark.gpu


def _state(n, flow, dscale=1.0, vscale=1.0, seed=3):
    ov = dict(ie=n[0], je=n[1], ke=n[2], gamma=1.4, courant=0.4, flux_limiter="minmod", t_end=1e60, dt_out=1e60,
              mag_on=False)
    for a in (1, 2, 3):
        for tag in ("is", "os", "iv", "ov"):
            ov[f"bc{a}{tag}"] = (3, 2, 1)[a - 1]
    cfg = config.resolve("riemann", overrides=ov)
    rng = np.random.default_rng(seed)
    shape = (n[2], n[1], n[0])
    z = np.zeros(shape)
    d = dscale * np.exp(rng.uniform(-1, 1, shape))
    cs = vscale
    p = d * cs * cs / 1.4 * rng.uniform(0.5, 1.5, shape)
    v = [z.copy() for _ in range(3)]
    if flow == "rest":  # pressure differences only; whole regions stay at rest
        p[:] = dscale * vscale * vscale
        p[..., : n[0] // 3] *= 2.0
        d[:] = dscale
    else:
        m = {"subsonic": 0.5, "right": 3.0, "left": -3.0}[flow]
        for a in range(3):
            v[a] = vscale * (m + 0.3 * rng.uniform(-1, 1, shape)) * (1.0 if n[a] > 1 else 0.0)
    return cfg, {"d": d, "p": p, "v1": v[0], "v2": v[1], "v3": v[2], "b1": z, "b2": z, "b3": z, "phi": z}


@pytest.mark.parametrize("n", [(37, 1, 1), (19, 18, 1), (17, 9, 7)])
@pytest.mark.parametrize("flow", ["rest", "subsonic", "right", "left"])
def test_flows(n, flow):
    run_pair(*_state(n, flow), 4)


# 2^-150 = 7e-46 and 2^200 = 1.6e60 bound the densities, 2^150 = 1.4e45 the
# speeds and 2^-200 = 6e-61 the wave distances of the short form
@pytest.mark.parametrize("dscale,vscale", [(7e-46, 1.0), (1e-47, 1.0), (1.6e60, 1.0), (1e62, 1.0), (1.0, 1.4e45),
                                           (1.0, 1e47), (1.0, 6e-61), (1.0, 1e-63), (1e-30, 1e20)])
def test_scales(dscale, vscale):
    run_pair(*_state((17, 9, 7), "subsonic", dscale, vscale), 2)
