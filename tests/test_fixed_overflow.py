"""The fixed-point collisions (lbm_fixed.cuh) keep to arithmetic that the language
defines: built for the host with the compiler's overflow and shift checks, over
accepted states up to the ends of the range, no sum, product or shift is
reported.  Runs without a GPU."""
import os
import shutil
import subprocess
import sys
import tempfile

import pytest

from test_device_math_host import _cuda_include
from test_fixed_math_host import MODELS

HERE = os.path.dirname(os.path.abspath(__file__))

DRIVER = """
import ctypes as C, sys
import numpy as np
sys.path[:0] = sys.argv[3:]
import lbmgpu as G
import test_fixed_math_host as T
lib, name, dp = C.CDLL(sys.argv[1]), sys.argv[2], C.POINTER(C.c_double)
n, rng = 400, np.random.default_rng(5)
out = [np.zeros(20 * 4000) for _ in range(6)]
o = [T.ptr(v) for v in out]
if name == "thermal":
    f, _ = T.states(T.model("d2q9_bgk"), n, 31, 0.08)
    t = np.ascontiguousarray(T.W5.astype(float) * (1 + rng.standard_normal((n, 5))))
    l, om = np.ascontiguousarray(rng.standard_normal((n, 5))), rng.uniform(0.05, 1.98, n)
    assert lib.fixed_thermal(n, T.ptr(f), T.ptr(t), T.ptr(l), T.ptr(om), *o[:5]) == n
else:
    cfg = T.model(name)
    c = cfg.to_c()
    for f, g in (T.states(cfg, n, 11, 0.08), T.corner_states(cfg, 5)):
        k = f.shape[0]
        assert lib.fixed_forward(C.byref(c), k, T.ptr(f), T.ptr(g), *o[:2]) == k
        for kind in ("rough", "spread"):
            lo = T.adjoints(cfg, k, kind)
            assert lib.fixed_reverse(C.byref(c), k, T.ptr(f), T.ptr(g), T.ptr(lo), *o[:4]) == k
        if cfg.lattice == G.D2Q9:
            s = C.c_int()
            d = cfg.replace(obj_weight=-3.0).to_c()
            assert lib.fixed_dissipation(C.byref(d), k, T.ptr(f), T.ptr(g), *o[:5],
                                         C.byref(s)) == k
print("done")
"""


@pytest.fixture(scope="module")
def checked_library():
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    so = os.path.join(tempfile.mkdtemp(), "libfixedchecked.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-ffp-contract=off",
                        "-fsanitize=signed-integer-overflow,shift", "-I" + inc,
                        os.path.join(HERE, "fixed_math_host.cpp"), "-o", so],
                       capture_output=True, text=True)
    if r.returncode and "ubsan" in r.stderr:
        pytest.skip("the compiler's check library is not installed")
    assert r.returncode == 0, r.stderr
    return so


@pytest.mark.parametrize("name", MODELS + ["thermal"])
def test_no_undefined_arithmetic(checked_library, name):
    r = subprocess.run([sys.executable, "-c", DRIVER, checked_library, name, HERE,
                        os.path.join(os.path.dirname(HERE), "lbm-topopt_gb300")],
                       capture_output=True, text=True)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr
    assert "runtime error" not in r.stderr, r.stderr
