"""One instance with few and very long lines: the tables of chunk products grow with the grid, not with the
square of the longer side, and the partitioned solves agree with the thread-per-line ones."""
import dataclasses

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(120000, 6), (6, 120000)])
@pytest.mark.parametrize("model", ["heston", "sabr"])
def test_device_memory_and_result(lss, nx, ny, model):
    import torch

    kw = dict(scheme="hv", nx=nx, ny=ny, nt=3, maturity=1e-6, rho=-0.2)
    if model == "sabr":  # coefficients that change with time
        kw.update(model="sabr", sabr_beta=0.5, sigma=0.4, rate=0.03, strike=0.05, s_hi=0.2, v_hi=1.0, eval_s=0.05, eval_v=0.3)
    p = lss.HestonProblem(**kw)
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    s = lss.ImplicitHestonSolver(p)
    free1, _ = torch.cuda.mem_get_info()
    # 5 states, 13 line tables, 6 arrays of time-dependent coefficients, products below the line tables,
    # up to 16 sets of the ten S tables with their products within 64 MB
    n = nx * ((ny + 3) // 4 * 4)
    assert free0 - free1 < 8 * n * 40 + (128 << 20)
    got, val = s.solve()
    ref, rval = lss.ImplicitHestonSolver(dataclasses.replace(p, line_per_thread=True)).solve()
    assert np.all(np.isfinite(ref))
    assert rel_err(got, ref) < 1e-9
    assert abs(val - rval) <= 1e-9 * max(1.0, abs(rval))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny", [(2600, 306), (2600, 308), (2600, 1218), (2600, 1220)])
def test_both_sides_of_the_lines_that_fill_the_gpu(lss, nx, ny, precision):
    """S lines of several tiles with 2, 4 and 8 lines per CTA: the split solves the thread-per-line systems."""
    p = lss.HestonProblem(scheme="hv", nx=nx, ny=ny, nt=3, maturity=1e-6, rho=-0.2)
    got, _ = lss.ImplicitHestonSolver(p, precision=precision).solve()
    ref, _ = lss.ImplicitHestonSolver(dataclasses.replace(p, line_per_thread=True), precision=precision).solve()
    assert np.all(np.isfinite(ref))
    assert rel_err(got, ref) < (1e-10 if precision == "f64" else 1e-4)
