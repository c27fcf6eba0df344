"""The factorised FP64 sweep in registers (k_h1_reg: W lanes of R rows per instance) at the sizes
where its split changes -- one row around every (lanes, rows) shape and around the last line that
fits -- for every boundary kind, both theta schemes, with and without a source, several instances
per warp with different step counts, against the CPU oracle."""
import numpy as np
import pytest

from conftest import rel_err
from test_heat1d_gpu import tables_problem

pytestmark = pytest.mark.gpu

SIZES = (4, 5, 15, 16, 17, 33, 63, 64, 65, 112, 127, 128, 129, 161, 224, 257, 320, 385, 449, 511, 512, 513)
ENDS = (("dirichlet", "dirichlet"), ("neumann", "robin"), ("robin", "dirichlet"), ("dirichlet", "neumann"))


@pytest.mark.parametrize("theta", ["cn", "euler"])
@pytest.mark.parametrize("lo,hi", ENDS)
@pytest.mark.parametrize("src", [False, True])
def test_register_sweep_at_every_shape(lss, oracle, theta, lo, hi, src):
    tabs, probs = [], []
    for n in SIZES:
        for nt in (2, 5, 9):
            kw = dict(model="const", x_hi=1.0, t_hi=0.2, n=n, nt=nt, forward=bool(nt == 5), lo_kind=lo, hi_kind=hi,
                      theta_scheme=theta, diff=0.7, conv=0.3, react=-0.2, init0=0.2, init1=1.0, lo_value=0.1,
                      hi_value=0.3, lo_linear=0.4 if lo == "robin" else 0.0, hi_linear=-0.5 if hi == "robin" else 0.0)
            if src:
                kw.update(has_source=True, src0=0.5, src1=-1.0)
            p, t = tables_problem(oracle, kw, "f64")
            probs.append(p)
            tabs.append(t)
    for every in (False, True):
        b = lss.tabulated_batch(tabs, "f64", "fast", all_steps=every)
        vals, st = b.run_host()
        assert not st.any()
        for i, p in enumerate(probs):
            want = oracle.solve_1d(p, "f64", all_steps=every)
            got = b.solution(i)
            assert got.shape == want.shape
            assert rel_err(got, want) < 1e-10, (p.n, p.nt)  # the path's stated FP64 tolerance
            last = got if not every else got[-1 if p.forward else 0]
            assert vals[i] == last[p.n // 2]


def test_register_sweep_repeats_bit_for_bit(lss):
    qs = lss.draw_black_scholes(70, seed=3)
    b = lss.black_scholes_batch(qs, "f64", "fast")
    v1, _ = b.run_host()
    v2, _ = b.run_host()
    assert np.array_equal(v1, v2)
