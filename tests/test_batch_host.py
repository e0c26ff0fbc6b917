"""Host side of the batch (hmn_batch.cu) without a GPU: tests/batch_host_check.cpp
compiles it against a made-up CUDA runtime in which a launch can fail."""
import os
import subprocess

from hormone_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_batch_host_logic(tmp_path):
    exe = str(tmp_path / "batch_host_check")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-x", "c++", "-std=c++17", "-O1", "-w", "-I", cuda, os.path.join(HERE, "batch_host_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
