"""The reference arithmetic with its factors made once (adi_exact.cuh): the same bits as the CPU oracle
at the sizes where the lines per CTA and the rows loaded ahead change, for terminal conditions whose
values leave the range of the division by a known divisor (zeros of either sign, denormal, tiny and huge
values), in both precisions and directly or as a graph.  Equality is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(lss, nx, ny, scheme, steps):
    slope = 1.2 / 24.0 * np.arcsinh(24.0)
    T = min(0.2, 0.5 * slope * steps / (1.5 * 0.04 * (ny - 1)))  # the explicit v = 0 line
    return lss.HestonProblem(scheme=scheme, rho=-0.3, maturity=float(T), nx=nx, ny=ny, nt=steps + 1, zeta=0.4, nonuniform=True,
                             acc_point=100.0, alpha_scale=10.0, beta_scale=24.0)


def same_bits(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    u = np.uint64 if a.dtype == np.float64 else np.uint32
    return a.dtype == b.dtype and np.array_equal(a.view(u), b.view(u))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 6), (6, 11), (10, 7), (11, 12), (154, 155), (155, 310), (610, 9), (9, 1300), (1500, 5)])
def test_bits_at_every_shape(lss, oracle, scheme, nx, ny, precision):
    p = problem(lss, nx, ny, scheme, 3)
    op = oracle.Problem(**p.pde_fields())
    want = oracle.solve(op, precision)
    s = lss.ImplicitHestonSolver(p, precision=precision, arith="reference")
    got, val = s.solve()
    assert same_bits(got, want)
    again, val2 = s.solve(graph=True)
    assert same_bits(again, want) and val == val2


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("scheme", ["dr", "mcs", "hv"])
def test_bits_outside_the_divisions_range(lss, oracle, scheme, precision):
    nx, ny = 60, 21
    p = problem(lss, nx, ny, scheme, 2)
    op = oracle.Problem(**p.pde_fields())
    t = np.float64 if precision == "f64" else np.float32
    rng = np.random.default_rng(3)
    big, small, sub = (1e290, 1e-290, 1e-310) if precision == "f64" else (1e30, 1e-32, 1e-40)
    for kind in ("zeros", "denormal", "tiny", "huge", "mixed"):
        pay = rng.standard_normal((nx, ny))
        if kind == "zeros":
            pay = np.where(rng.random((nx, ny)) < 0.5, -0.0, 0.0)
        elif kind == "denormal":
            pay *= sub
        elif kind == "tiny":
            pay *= small
        elif kind == "huge":
            pay *= big
        else:
            pay *= np.where(rng.random((nx, ny)) < 0.3, small, 1.0)
            pay[::7] = -0.0
        pay = pay.astype(t)
        want = oracle.solve(op, precision, payoff=pay)
        got, _ = lss.ImplicitHestonSolver(p, precision=precision, arith="reference").solve(payoff=pay)
        assert same_bits(got, want), kind
