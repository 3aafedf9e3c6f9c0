"""Arrays crossing the C ABI: designs and design variables are refused on the
device as on the host (sizes around the 8192 values from which the check runs
there), with the old ones kept; results come out the same in fresh, reused and
oddly placed host memory (large arrays get their pages first)."""
import ctypes as C

import numpy as np
import pytest

import lbmgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(127, 64), (128, 64), (129, 64), (300, 200)])
@pytest.mark.parametrize("value,code", [(-1e-12, G.ERR_ARG), (1.0 + 1e-12, G.ERR_ARG),
                                        (np.nan, G.ERR_NONFINITE), (np.inf, G.ERR_NONFINITE)])
def test_bad_designs_are_refused_and_the_old_one_kept(nx, ny, value, code):
    cfg = W.channel_2d(nx, ny, nsteps=5)
    gamma = W.design_2d(nx, ny, 3)
    gamma[:2] = 0.0, 1.0
    with G.Handle(cfg) as h:
        h.set_design(gamma)
        J, s, _ = h.gradient(5, 3)
        for i in (0, 1, nx * ny // 2, nx * ny - 1):
            bad = gamma.copy()
            bad[i] = value
            with pytest.raises(G.LBMError) as e:
                h.set_design(bad)
            assert e.value.code == code and str(i) in str(e.value)
        J2, s2, _ = h.gradient(5, 3)
    assert J == J2 and np.array_equal(s, s2)


@pytest.mark.parametrize("n", [5, 300, 80001])
@pytest.mark.parametrize("value", [-1e-12, 1.0 + 1e-12, np.nan])
def test_bad_variables_are_refused_and_the_old_ones_kept(n, value):
    x = np.random.default_rng(1).uniform(0, 1, n)
    with G.TopOpt(n, 1, 1, (0, n - 1, 0, 0, 0, 0), stages=(), x0=x) as t:
        for i in (0, n - 1):
            bad = x.copy()
            bad[i] = value
            with pytest.raises(G.LBMError) as e:
                t.set_variables(bad)
            assert e.value.code == G.ERR_ARG and str(i) in str(e.value)
            assert np.array_equal(t.variables(), x)
        y = x[::-1].copy()
        y[0], y[-1] = 0.0, 1.0
        t.set_variables(y)
        assert np.array_equal(t.variables(), y)


@pytest.mark.parametrize("nx,ny", [(40, 30), (121, 121), (640, 200)])
def test_results_in_any_host_memory(nx, ny):
    cfg = W.channel_2d(nx, ny, nsteps=3)
    with G.Handle(cfg) as h:
        h.set_design(W.design_2d(nx, ny, 3))
        h.init_equilibrium()
        h.forward(3)
        f = h.populations()
        n = f.size
        keep = np.full(n + 3, 7.0)
        for off in (0, 1, 3):
            keep[:] = 7.0
            p = C.cast(keep.ctypes.data + 8 * off, C.POINTER(C.c_double))
            h._check(h.lib.lbm_get_populations(h.h, p))
            assert np.array_equal(keep[off:off + n], f)
            assert (keep[:off] == 7.0).all() and (keep[off + n:] == 7.0).all()


def test_results_of_many_handles_in_threads():
    """Handles share pages of 64 result slots: more than two pages' worth alive at
    once, used from four threads, closed and made again."""
    import threading
    import workloads as W
    cfg = W.channel_2d(20, 12, nsteps=4)
    designs = [W.design_2d(20, 12, 50 + k) for k in range(140)]

    def value(h, k):
        h.set_design(designs[k])
        h.init_equilibrium()
        return h.forward(4)
    with G.Handle(cfg) as h:
        want = [value(h, k) for k in range(140)]
    got = [[None] * 140 for _ in range(2)]

    def work(part):
        for turn in range(2):
            hs = {k: G.Handle(cfg) for k in range(part, 140, 4)}
            for k, x in hs.items():
                got[turn][k] = value(x, k)
            for x in hs.values():
                x.close()
    threads = [threading.Thread(target=work, args=(p,)) for p in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got[0] == want and got[1] == want
