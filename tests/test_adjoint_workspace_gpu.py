"""The workspace of a single instance's adjoint: bounded when the interval is planned, usable again after an
allocation that failed, kept from call to call, and free of traces of the call before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NU = dict(nonuniform=True, acc_point=100.0, alpha_scale=10.0, beta_scale=24.0)


def same(a, b):
    return a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])


def test_planned_workspace_is_bounded_and_kept(lss):
    import torch

    # every step kept: 4 arrays of 1000 x 500 points times 1600 steps, 25.6 GB
    p = lss.HestonProblem(nx=1000, ny=500, nt=1601, maturity=0.05, rho=-0.2, **NU)
    s = lss.ImplicitHestonSolver(p)
    torch.cuda.synchronize()
    free0, total = torch.cuda.mem_get_info()
    assert 25.6e9 > total / 16
    first = s.adjoint()
    free1, _ = torch.cuda.mem_get_info()
    assert free0 - free1 < total / 16 + (1 << 30)  # (tables of half a million points besides)
    hold = torch.empty(int(0.9 * free1), dtype=torch.uint8, device="cuda")
    free2, _ = torch.cuda.mem_get_info()
    again = s.adjoint()
    assert torch.cuda.mem_get_info()[0] == free2  # no other interval because others hold memory
    assert same(first, again)
    del hold
    torch.cuda.empty_cache()


def test_a_failed_allocation_leaves_the_handle_usable(lss):
    import torch
    from linear_system_solvers_gb300 import _lib as L

    p = lss.HestonProblem(nx=512, ny=256, nt=201, maturity=0.1, rho=-0.2, scheme="cs", **NU)
    s = lss.ImplicitHestonSolver(p)
    want = s.adjoint(checkpoint_every=15)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (600 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(L.LssError) as err:
            s.adjoint(checkpoint_every=200)  # 843 MB
        assert err.value.code == L.ENOMEM
        assert same(s.adjoint(checkpoint_every=15), want)
        assert same(s.adjoint(), want)  # planned within what is free
    finally:
        del hold
        torch.cuda.empty_cache()


@pytest.mark.parametrize("scheme", ["dr", "cs", "mcs", "hv"])
@pytest.mark.parametrize("kw", [dict(nx=37, ny=18), dict(nx=37, ny=18, wide_adjoint=True), dict(nx=1031, ny=9),
                                dict(nx=9, ny=1027, wide_adjoint=True)])
def test_nothing_of_the_call_before_is_read(lss, scheme, kw):
    p = lss.HestonProblem(scheme=scheme, nt=12, maturity=0.002, rho=-0.2, zeta=1.0 / 3.0, **kw, **NU)
    pay = np.random.default_rng(1).uniform(0.0, 50.0, (p.nx, p.ny))
    for ck in (0, 3, 11):
        fresh = lss.ImplicitHestonSolver(p).adjoint(payoff=pay, checkpoint_every=ck)
        s = lss.ImplicitHestonSolver(p)
        bad = s.adjoint(payoff=np.full_like(pay, np.nan), checkpoint_every=ck)
        assert np.isnan(bad[0])
        assert np.all(np.isfinite(fresh[2])) and same(s.adjoint(payoff=pay, checkpoint_every=ck), fresh)
