"""The partitioned line solves of one instance (adi_wide.cuh) at the sizes where their split changes:
lines that end just before, on and just after a chunk, the longest lines of 5, 8 and 16 rows per S
chunk and of 4, 8 and 16 per v chunk, lines of several tiles, odd row pitches, and the smallest
grid; forward against the thread-per-line solve and the CPU oracle, the adjoint against the same
kernels with one chunk per line (dV/d(payoff) and the sensitivities are sums over the same terms in
another order).  On these stretched grids (k / h^2 up to 1e6) the reference scheme itself amplifies
rounding, so the forward bound is that of the other partition tests: 100x the spread that a 1e-15
relative perturbation of the terminal condition causes in the oracle (floor 1e-13; 1e-10 against
the oracle)."""
import dataclasses

import numpy as np
import pytest

from conftest import fp64_tol, fp32_ok, rel_err

pytestmark = pytest.mark.gpu

NU = dict(nonuniform=True, acc_point=100.0, alpha_scale=10.0, beta_scale=24.0)
S_SIZES = (4, 5, 6, 7, 11, 12, 13, 641, 642, 643, 1025, 1026, 1027, 2049, 2050, 2051, 2600)
V_SIZES = (4, 5, 7, 8, 9, 15, 16, 17, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1300)


def problem(lss, nx, ny, scheme, steps=3, **kw):
    # the explicit v = 0 line: Courant number kappa theta k / (2 h2 B(0)) of at most 0.25
    slope = 1.2 / 24.0 * np.arcsinh(24.0)
    T = min(0.2, 0.5 * slope * steps / (1.5 * 0.04 * (ny - 1)))
    return lss.HestonProblem(scheme=scheme, rho=-0.2, maturity=float(T), nx=nx, ny=ny, nt=steps + 1, zeta=1.0 / 3.0, **NU, **kw)


def oracle_of(oracle, p):
    return oracle.Problem(**p.pde_fields())


@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
@pytest.mark.parametrize("nx,ny", [(n, 9) for n in S_SIZES] + [(10, n) for n in V_SIZES])
def test_forward_at_every_split(lss, oracle, scheme, nx, ny):
    p = problem(lss, nx, ny, scheme)
    op = oracle_of(oracle, p)
    want = oracle.solve(op, "f64")
    x, _ = oracle.grid(op, "f64")
    pay = np.maximum(x[:, None] - p.strike, 0.0) * np.ones((1, ny))
    noisy = pay * (1.0 + 1e-15 * np.random.default_rng(1).standard_normal(pay.shape))
    amp = rel_err(oracle.solve(op, "f64", payoff=noisy), want)
    ref, rval = lss.ImplicitHestonSolver(dataclasses.replace(p, line_per_thread=True)).solve()
    s = lss.ImplicitHestonSolver(p)
    got, val = s.solve()
    tol = max(1e-13, 100.0 * amp)
    assert rel_err(got, ref) < tol
    assert abs(val - rval) <= tol * max(1.0, abs(rval))
    assert rel_err(got, want) < max(fp64_tol(want, p.s_hi), tol)
    again, val2 = s.solve(graph=True)
    assert np.array_equal(got, again) and val == val2


@pytest.mark.parametrize("nx,ny", [(6, 5), (643, 257), (1027, 18), (2051, 9), (11, 1025)])
def test_forward_fp32_at_every_split(lss, oracle, nx, ny):
    p = problem(lss, nx, ny, "hv")
    op = oracle_of(oracle, p)
    got, _ = lss.ImplicitHestonSolver(p, precision="f32").solve()
    ok, e_dev, e_ref = fp32_ok(got, oracle.solve(op, "f32"), oracle.solve(op, "f64"))
    assert ok, (e_dev, e_ref)


@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 9), (13, 17), (642, 9), (643, 14), (1027, 8), (2051, 9), (2600, 6), (10, 256),
                                   (9, 257), (8, 513), (12, 1025), (6, 1300)])
def test_adjoint_at_every_split(lss, scheme, nx, ny):
    p = problem(lss, nx, ny, scheme, wide_adjoint=True)
    val, g, lam = lss.ImplicitHestonSolver(p).adjoint()
    one = lss.ImplicitHestonSolver(dataclasses.replace(p, line_per_thread=True))
    v1, g1, lam1 = one.adjoint()
    assert abs(val - v1) <= 1e-11 * max(1.0, abs(v1))
    assert np.max(np.abs(g - g1)) <= 1e-9 * max(np.abs(g1).max(), 1e-3 * abs(v1))
    assert np.max(np.abs(lam - lam1)) <= 1e-9 * np.abs(lam1).max()
    # the adjoint is the exact linear response of the forward pass
    s = lss.ImplicitHestonSolver(p)
    x, _ = s.grid()
    pay = np.repeat(np.maximum(x - p.strike, 0.0)[:, None], ny, axis=1)
    delta = np.random.default_rng(2).normal(size=pay.shape)
    resp = s.solve(payoff=pay + delta)[1] - s.solve(payoff=pay)[1]
    assert abs(resp - float(np.sum(lam * delta))) <= 1e-9 * max(1.0, np.sum(np.abs(lam * delta)))


def test_adjoint_time_dependent_segments(lss):
    """SABR with r != 0 on the partitioned kernels: the refactorised tables of every step serve the
    forward pass, the recomputation of a segment and the adjoint alike (bitwise the same results
    for every checkpoint interval)."""
    p = lss.HestonProblem(model="sabr", sabr_beta=0.5, sigma=0.4, rho=-0.3, rate=0.03, strike=0.05, maturity=1.0, s_lo=0.0,
                          s_hi=0.2, v_lo=0.0, v_hi=1.0, nx=90, ny=43, nt=14, scheme="hv", nonuniform=True, acc_point=0.05,
                          alpha_scale=3.0, beta_scale=5.0, eval_s=0.05, eval_v=0.3)
    s = lss.ImplicitHestonSolver(p)
    ref = s.adjoint()
    for ck in (1, 4, 13):
        got = s.adjoint(checkpoint_every=ck)
        assert got[0] == ref[0] and np.array_equal(got[1], ref[1]) and np.array_equal(got[2], ref[2])
