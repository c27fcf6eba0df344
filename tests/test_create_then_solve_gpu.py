"""A solver is ready when its creation returns: the first solve of a new handle, queued at once on a
non-blocking stream with device pointers (nothing orders that stream behind the default stream on
which the set-up ran), has the bits of a later solve of the same handle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NU = dict(nonuniform=True, acc_point=100.0, alpha_scale=10.0, beta_scale=24.0)
SABR_T = dict(model="sabr", sabr_beta=0.5, sigma=0.4, rho=-0.3, rate=0.03, strike=0.05, maturity=0.2, s_lo=0.0, s_hi=0.2, v_lo=0.0,
              v_hi=1.0, nonuniform=True, acc_point=0.05, alpha_scale=3.0, beta_scale=5.0, eval_s=0.05, eval_v=0.3)
CASES = {
    "dr_small": (dict(nx=40, ny=20, nt=4, **NU), "f64"),
    "hv_tiles": (dict(nx=4096, ny=1300, nt=3, maturity=0.01, scheme="hv", **NU), "f64"),
    "cs_tiles_f32": (dict(nx=4096, ny=1300, nt=3, maturity=0.01, scheme="cs", **NU), "f32"),
    "sabr_t": (dict(SABR_T, nx=900, ny=700, nt=4, scheme="hv"), "f64"),
    "sabr_t_groups": (dict(SABR_T, nx=64, ny=40, nt=40, scheme="dr"), "f64"),
}


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("key", sorted(CASES))
def test_first_solve_on_a_non_blocking_stream(lss, key, graph):
    import torch

    from linear_system_solvers_gb300 import _lib as L

    kw, fp = CASES[key]
    p = lss.HestonProblem(**kw)
    dt = torch.float32 if fp == "f32" else torch.float64
    side = torch.cuda.Stream()
    lib = L.load()
    with torch.cuda.stream(side):
        pay = torch.rand(p.nx, p.ny, dtype=dt, device="cuda")
        first, second = torch.zeros_like(pay), torch.zeros_like(pay)
    torch.cuda.synchronize()
    fn = lib.lss_adi_forward_graph if graph else lib.lss_adi_forward
    for _ in range(3):
        s = lss.ImplicitHestonSolver(p, precision=fp)
        for out in (first, second):
            L.check(fn(s._h, pay.data_ptr(), out.data_ptr(), None, L.DEVICE_POINTERS, ctypes.c_void_p(side.cuda_stream)))
            if out is first:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        a, b = first.cpu().numpy(), second.cpu().numpy()
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)
        s.close()
