"""The adjoint of one instance where its route changes: relay order (the recurrences over the chunks one
after the other) has the bits of the same instance in a batch at every split, and the S-line tables
of time-dependent coefficients, made for several steps by one launch, at the splits of the S lines
and at step counts around the size of a group.  Equalities are exact; the comparison with the CPU
oracle has the bound of the other partition tests (100x the spread that a 1e-15 relative
perturbation of the terminal condition causes in the oracle, floor 1e-13; 1e-10 against the oracle)."""
import dataclasses

import numpy as np
import pytest

from conftest import fp64_tol, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
@pytest.mark.parametrize("nx,ny", [(4, 4), (7, 9), (43, 17), (100, 50), (129, 66), (256, 130)])
def test_relay_order_has_the_bits_of_a_batch(lss, scheme, nx, ny):
    p = lss.HestonProblem(scheme=scheme, rho=-0.4, maturity=0.02, nx=nx, ny=ny, nt=5, zeta=0.4, alpha_scale=3.0, beta_scale=8.0,
                          nonuniform=True, acc_point=100.0)
    val, g, lam = lss.ImplicitHestonSolver(p).adjoint()
    b = lss.BatchSolver([p])
    b.run(1)
    values, grads, _ = b.results()
    assert val == values[0]
    np.testing.assert_allclose(g, grads[0], rtol=0, atol=1e-12 * max(np.abs(g).max(), abs(val)))


@pytest.mark.parametrize("scheme", ["dr", "mcs", "hv"])
@pytest.mark.parametrize("nx,ny,steps", [(4, 4, 3), (9, 6, 16), (43, 21, 17), (643, 14, 5), (1027, 8, 4), (2051, 9, 3), (90, 43, 33)])
def test_time_dependent_tables_in_groups(lss, oracle, scheme, nx, ny, steps):
    p = lss.HestonProblem(model="sabr", sabr_beta=0.5, sigma=0.4, rho=-0.3, rate=0.03, strike=0.05, maturity=0.1, s_lo=0.0,
                          s_hi=0.2, v_lo=0.0, v_hi=1.0, nx=nx, ny=ny, nt=steps + 1, scheme=scheme, nonuniform=True, acc_point=0.05,
                          alpha_scale=3.0, beta_scale=5.0, eval_s=0.05, eval_v=0.3, wide_adjoint=True)
    op = oracle.Problem(**p.pde_fields())
    want = oracle.solve(op, "f64")
    x, _ = oracle.grid(op, "f64")
    pay = np.maximum(x[:, None] - p.strike, 0.0) * np.ones((1, ny))
    noisy = pay * (1.0 + 1e-15 * np.random.default_rng(1).standard_normal(pay.shape))
    tol = max(1e-13, 100.0 * rel_err(oracle.solve(op, "f64", payoff=noisy), want))
    s = lss.ImplicitHestonSolver(p)
    got, val = s.solve()
    assert rel_err(got, want) < max(fp64_tol(want, p.s_hi), tol)
    again, val2 = s.solve(graph=True)
    assert np.array_equal(got, again) and val == val2
    ref = s.adjoint()
    assert ref[0] == val
    for ck in (1, max(1, steps // 2)):
        new = s.adjoint(checkpoint_every=ck)
        assert new[0] == ref[0] and np.array_equal(new[1], ref[1]) and np.array_equal(new[2], ref[2])
    # the adjoint is the exact linear response of the forward pass
    delta = np.random.default_rng(2).normal(size=pay.shape)
    resp = s.solve(payoff=pay + delta)[1] - s.solve(payoff=pay)[1]
    assert abs(resp - float(np.sum(ref[2] * delta))) <= 1e-9 * max(1.0, np.sum(np.abs(ref[2] * delta)))
