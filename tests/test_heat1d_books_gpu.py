"""FP64 books of many short lines run the sweep through memory, smaller books the sweep in registers
(memory_limit): the same systems, so the same values to rounding, also where a book mixes both; and the
shapes of the sweeps in registers follow the rows that an instance solves, not its points."""
import numpy as np
import pytest

from conftest import rel_err
from test_heat1d_gpu import bs_oracle_problem, tables_problem

pytestmark = pytest.mark.gpu


def book(lss, n, count, nt=12):
    r = np.random.default_rng(n)
    return [lss.BlackScholesProblem(sigma=float(r.uniform(0.15, 0.4)), rate=0.03, strike=10.0, maturity=float(r.uniform(0.5, 1.5)), s_lo=0.0,
                                    s_hi=40.0, n=n, nt=nt, theta_scheme="cn" if k % 2 else "euler", nonuniform=True, acc_point=10.0,
                                    alpha_scale=3.0, eval_s=10.0) for k in range(count)]


@pytest.mark.parametrize("n", [4, 9, 50, 100])
def test_a_large_book_has_the_values_of_small_ones(lss, oracle, n):
    qs = book(lss, n, 60000)
    large = lss.black_scholes_batch(qs, "f64")
    v, st = large.run_host()
    small = lss.black_scholes_batch(qs[:64], "f64")
    w, _ = small.run_host()
    assert not st.any() and np.max(np.abs(v[:64] - w)) <= 1e-12 * np.max(np.abs(w))
    for i in (0, 1, 63, 59999):
        assert rel_err(large.solution(i), oracle.solve_1d(bs_oracle_problem(oracle, qs[i]), "f64")) < 1e-10
    mixed = lss.black_scholes_batch(qs + book(lss, 300, 40), "f64")
    m, st = mixed.run_host()
    assert not st.any() and np.max(np.abs(m[:64] - w)) <= 1e-12 * np.max(np.abs(w))
    if mixed.launch_count() == 2:  # the short lines kept their sweep
        assert np.array_equal(m[:64], v[:64])
    else:
        assert np.array_equal(m[:64], w)


@pytest.mark.parametrize("lo,hi", [("dirichlet", "dirichlet"), ("neumann", "dirichlet"), ("robin", "neumann")])
@pytest.mark.parametrize("n", [17, 18, 64, 65, 66, 128, 129, 130, 193, 194, 256, 257, 258, 510, 512])
def test_every_number_of_solved_rows(lss, oracle, n, lo, hi):
    kw = dict(model="const", x_hi=1.0, t_hi=0.2, n=n, nt=7, lo_kind=lo, hi_kind=hi, theta_scheme="cn", diff=0.7, conv=0.3, react=-0.2, init0=0.2,
              init1=1.0, lo_value=0.1, hi_value=0.3, lo_linear=0.4 if lo == "robin" else 0.0)
    p, t = tables_problem(oracle, kw, "f64")
    b = lss.tabulated_batch([t] * 3, "f64", "fast")
    b.run_host()
    assert rel_err(b.solution(2), oracle.solve_1d(p, "f64")) < 1e-10


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_both_sweeps_of_a_book_end_with_the_run(lss, precision):
    """Lines for both sweeps in one book, which run beside each other: runs that follow at once on the same
    stream, and a read of the results queued behind them, see the values of each sweep alone."""
    short, long_lines = book(lss, 500, 400, nt=40), book(lss, 700, 30, nt=40)
    b = lss.black_scholes_batch(short + long_lines, precision)
    assert b.launch_count() == 2
    want = np.concatenate([lss.black_scholes_batch(q, precision).run_host()[0] for q in (short, long_lines)])
    for _ in range(20):
        for _ in range(3):
            b.run()
        v, st = b.results()
        assert not st.any() and np.array_equal(v, want)
