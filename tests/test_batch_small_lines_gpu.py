"""Batches of small grids run kernels that load fewer rows ahead: on both sides of the sizes at which they are
chosen (256 points in FP32, 900 in FP64) a batch has the bits of the thread-per-line solve of its
instances, and a batch that mixes small and large ones too."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NU = dict(nonuniform=True, acc_point=100.0, alpha_scale=10.0, beta_scale=24.0)
SIZES = [(4, 4), (5, 4), (4, 7), (8, 8), (16, 16), (16, 17), (18, 15), (64, 4), (4, 64), (30, 30), (31, 30), (9, 100), (100, 9), (12, 75), (13, 75)]


def problem(lss, scheme, nx, ny, steps=7):
    return lss.HestonProblem(scheme=scheme, nx=nx, ny=ny, nt=steps + 1, maturity=0.01, rho=-0.3, zeta=0.4, **NU)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
def test_bits_of_the_thread_per_line_solve(lss, scheme, precision):
    ps = [problem(lss, scheme, nx, ny, 5 + k % 3) for k, (nx, ny) in enumerate(SIZES)]
    want = [lss.ImplicitHestonSolver(dataclasses.replace(p, line_per_thread=True), precision=precision).solve() for p in ps]
    large = problem(lss, scheme, 60, 40)
    for p, w in zip(ps, want):
        for batch in ([p] * 3, [p, large]):
            b = lss.BatchSolver(batch, precision=precision)
            b.run(0)
            assert np.array_equal(b.surface(0), w[0]), (p.nx, p.ny, len(batch))
            assert b.results()[0][0] == w[1] and not b.results()[2].any()
    mixed = lss.BatchSolver(ps + [large], precision=precision)
    mixed.run(0, graph=True)
    for k, w in enumerate(want):
        assert np.array_equal(mixed.surface(k), w[0])
