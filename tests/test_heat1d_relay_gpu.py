"""The FP32 factorised sweep in registers (k_h1_relay) has the values of the sweep through memory, which
instances take when one of their size in the batch has a source: one row around every (lanes, rows)
shape, every boundary kind, both theta schemes and directions, several step counts per warp, last
level and all levels.  Equality is exact."""
import numpy as np
import pytest

from test_heat1d_gpu import tables_problem

pytestmark = pytest.mark.gpu

SIZES = (4, 7, 8, 9, 15, 16, 17, 33, 64, 65, 112, 127, 128, 129, 161, 224, 257, 320, 385, 449, 511, 512, 513)
ENDS = (("dirichlet", "dirichlet"), ("neumann", "robin"), ("robin", "dirichlet"), ("dirichlet", "neumann"))


@pytest.mark.parametrize("theta", ["cn", "euler"])
@pytest.mark.parametrize("lo,hi", ENDS)
def test_relay_has_the_values_of_the_sweep_through_memory(lss, oracle, theta, lo, hi):
    tabs, extra = [], []
    for n in SIZES:
        kw = dict(model="const", x_hi=1.0, t_hi=0.2, n=n, lo_kind=lo, hi_kind=hi, theta_scheme=theta, diff=0.7, conv=0.3,
                  react=-0.2, init0=0.2, init1=1.0, lo_value=0.1, hi_value=0.3, lo_linear=0.4 if lo == "robin" else 0.0,
                  hi_linear=-0.5 if hi == "robin" else 0.0)
        for nt in (2, 5, 9, 12, 30):
            tabs.append(tables_problem(oracle, dict(kw, nt=nt, forward=bool(nt % 2)), "f32")[1])
        extra.append(tables_problem(oracle, dict(kw, nt=3, forward=True, has_source=True, src0=0.5, src1=-1.0), "f32")[1])
    for every in (False, True):
        b = lss.tabulated_batch(tabs, "f32", "fast", all_steps=every)
        vals, st = b.run_host()
        m = lss.tabulated_batch(tabs + extra, "f32", "fast", all_steps=every)
        want, wst = m.run_host()
        assert not st.any() and not wst.any()
        assert np.array_equal(vals, want[:len(tabs)])
        for i, t in enumerate(tabs):
            assert np.array_equal(b.solution(i), m.solution(i)), (t["n"], t["nt"])
