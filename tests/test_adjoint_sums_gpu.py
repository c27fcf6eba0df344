"""Gradients of a small instance against those of the same instance in a batch.

The parameter sums of an adjoint in relay order are made with the operations of the batched kernel in its
order.  An instance of at most 130 v points runs in a batch on a warp group with a thread per line, and the
gradients come out with the same bits, whatever the checkpoint interval; also where the scheme has growing
modes, whose sums are small against their terms (a call of 40 x 20 points was 1.05e-13 apart).
"""
import numpy as np
import pytest

import linear_system_solvers_gb300 as lss
from linear_system_solvers_gb300.batch import draw_batch

pytestmark = pytest.mark.gpu


def same(probs, **kw):
    bt = lss.BatchSolver(probs, precision="f64")
    bt.run(mode=1)
    values, grads, status = bt.results()
    for k, p in enumerate(probs):
        v, g, lam = lss.ImplicitHestonSolver(p, precision="f64", arith="fast").adjoint(**kw)
        assert v == values[k] or (np.isnan(v) and np.isnan(values[k]))
        assert np.array_equal(lam, bt.payoff_gradient(k), equal_nan=True)
        assert np.array_equal(g, grads[k], equal_nan=True), (k, g, grads[k])


@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
def test_heston_gradients_have_the_bits_of_the_batch(scheme):
    for seed in (7, 11, 31):
        probs = draw_batch(4, seed=seed)
        for k, p in enumerate(probs):
            p.scheme = scheme
            p.nx, p.ny, p.nt = (40, 48, 56, 64)[k], (20, 24, 28, 32)[k], 16 + 3 * k
        same(probs)


def test_genuine_modified_scheme():
    probs = draw_batch(3, seed=5)
    for k, p in enumerate(probs):
        p.nx, p.ny, p.nt = (24, 33, 70)[k], (16, 34, 21)[k], 6 + k
        p.zeta = 1.0 / 3.0
    same(probs)


@pytest.mark.parametrize("nx, ny, nt", [(4, 4, 3), (5, 34, 9), (7, 35, 8), (200, 66, 12), (256, 130, 4), (100, 129, 6)])
@pytest.mark.parametrize("scheme", ["dr", "cs", "hv"])
def test_edges_of_warps_and_rows(nx, ny, nt, scheme):
    same([lss.HestonProblem(nx=nx, ny=ny, nt=nt, scheme=scheme, rho=-0.2, nonuniform=True, acc_point=100.0,
                            alpha_scale=10.0, beta_scale=24.0)])


@pytest.mark.parametrize("every", [0, 7, 40])
@pytest.mark.parametrize("scheme", ["dr", "cs", "hv"])
def test_sabr_gradients_have_the_bits_of_the_batch(scheme, every):
    """Their terms hold the time of the step, in segments of any length."""
    same([lss.HestonProblem(model="sabr", sigma=0.4, rho=-0.3, sabr_beta=0.5, rate=0.0, strike=0.05, maturity=2.0, s_lo=0.0,
                            s_hi=0.2, v_lo=0.0, v_hi=1.0, nx=60, ny=40, nt=75, scheme=scheme, nonuniform=True, acc_point=0.05,
                            alpha_scale=10.0, beta_scale=24.0, eval_s=0.05, eval_v=0.2)], checkpoint_every=every)


@pytest.mark.parametrize("every", [1, 4, 19, 20, 50])
def test_checkpoint_interval_changes_no_bit(every):
    probs = draw_batch(1, seed=7)
    probs[0].nx, probs[0].ny, probs[0].nt = 40, 20, 21
    same(probs, checkpoint_every=every)


def test_line_per_thread_of_more_lines_than_a_group_has_threads():
    """A thread of the batch's group has several lines then: the order of the sums is still the batch's."""
    p = lss.HestonProblem(nx=300, ny=280, nt=5, scheme="cs", rho=-0.2, nonuniform=True, acc_point=100.0, alpha_scale=10.0,
                          beta_scale=24.0, line_per_thread=True)
    same([p])


def test_more_steps_than_a_run():
    """300 x 300 points: runs of 93 steps."""
    p = lss.HestonProblem(nx=300, ny=300, nt=121, maturity=0.2, scheme="dr", rho=-0.2, nonuniform=True, acc_point=100.0,
                          alpha_scale=10.0, beta_scale=24.0, line_per_thread=True)
    same([p])
    same([p], checkpoint_every=100)
