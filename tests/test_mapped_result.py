"""The mapped host memory of a handle's results, over a fake CUDA runtime: a
failed call leaves nothing half taken, and nothing is shared between handles or
outlives them.  Runs without a GPU."""
import os
import shutil
import subprocess

import pytest

from test_device_math_host import _cuda_include

HERE = os.path.dirname(os.path.abspath(__file__))


def test_take_and_give(tmp_path):
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "mapped_result_sim")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + inc, "-I",
                           os.path.join(os.path.dirname(HERE), "lbm-topopt_gb300", "csrc"),
                           os.path.join(HERE, "mapped_result_sim.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
