"""The quotients, reciprocals and square roots that the FP64 stages form
(hormone_b200/csrc/hmn_div.cuh, FastDiv) against the IEEE operations on the
GPU: tests/fastdiv_check.cu, compiled here with the library's FP64 flags,
requires every result that is not flagged to have the same bits, over operands
at the edges of the range, next to rounding midpoints and with zero numerators
of either sign.  A flagged result is recomputed with IEEE operations by the
stages, so this is what their bitwise parity rests on."""
import os
import subprocess

import pytest

from hormone_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_unflagged_results_are_the_ieee_ones(tmp_path):
    exe = str(tmp_path / "fastdiv_check")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-I", build.CSRC,
                    os.path.join(HERE, "fastdiv_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe, str(1 << 24), "20261203"], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
    stats = {l.split()[0]: dict(kv.split("=") for kv in l.split()[1:]) for l in r.stdout.splitlines() if " n=" in l}
    assert len(stats) == 12 and all(int(s["mismatches"]) == 0 for s in stats.values()), stats
    # operands inside the range are hardly ever flagged
    for fam in ("div_runs", "div_zero", "div_midpoints", "sqrt_squares", "sqrt_closest"):
        assert int(stats[fam]["flagged"]) <= int(stats[fam]["n"]) // 20, (fam, stats[fam])
