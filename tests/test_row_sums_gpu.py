"""Row sums of the explicit operator along v: with lines so fine that the weights W of a v line are large,
rounding a weight is worth eps W of the surface.  Such roundings must not add up over the steps: the result
stays within eps max(W) of the oracle for any number of steps."""
import dataclasses

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
SABR = dict(model="sabr", sabr_beta=0.5, sigma=0.4, rho=-0.3, strike=0.05, maturity=0.5, s_lo=0.0, s_hi=0.2, v_lo=0.0, v_hi=1.0,
            nonuniform=True, acc_point=0.05, alpha_scale=3.0, beta_scale=5.0, eval_s=0.05, eval_v=0.3)
# a slow drift keeps the explicit v = 0 line stable at large steps
HESTON = dict(kappa=0.01, theta_v=0.01, sigma=0.5, rho=-0.3, strike=100.0, maturity=1.0, nonuniform=True, acc_point=100.0, alpha_scale=10.0,
              beta_scale=5.0)


@pytest.mark.parametrize("rate", [1e-9, 0.03])
@pytest.mark.parametrize("model", ["sabr", "heston"])
def test_roundings_of_the_weights_do_not_add_up(lss, oracle, model, rate):
    p = lss.HestonProblem(nx=12, ny=3000, nt=11, scheme="dr", rate=rate, **(SABR if model == "sabr" else HESTON))
    op = oracle.Problem(**p.pde_fields())
    want = oracle.solve(op, "f64")
    bound = EPS * oracle.coefficients(op, 0.0)["W"].max()
    assert bound > 5e-13
    got, val = lss.ImplicitHestonSolver(p).solve()
    assert rel_err(got, want) < bound
    relay, _ = lss.ImplicitHestonSolver(dataclasses.replace(p, line_per_thread=True)).solve()
    assert rel_err(relay, want) < bound
    assert abs(lss.ImplicitHestonSolver(p).adjoint()[0] - val) < bound * max(1.0, abs(val))
    if model == "heston":
        b = lss.BatchSolver([p])
        for mode in (0, 1):
            b.run(mode)
            assert rel_err(b.surface(0), want) < bound
