"""Chunk counts set with lss_adi_line_chunks and the adjoint of the same handle."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["heston", "sabr_t"])
@pytest.mark.parametrize("adjoint_first", [False, True])
def test_set_chunk_counts_reach_the_adjoint_of_a_thread_per_line_handle(lss, model, adjoint_first):
    """lss_adi_line_chunks makes a LINE_PER_THREAD handle a partitioned one: forward solve and adjoint (of an
    instance too large for the batched order) solve the same partition, so the value has the same bits."""
    kw = dict(nx=300, ny=90, nt=9, maturity=0.01, scheme="cs", rho=-0.2, line_per_thread=True)
    if model == "sabr_t":
        kw.update(model="sabr", sabr_beta=0.5, sigma=0.4, rate=0.03, strike=0.05, s_hi=0.2, v_hi=1.0, eval_s=0.05, eval_v=0.3)
    p = lss.HestonProblem(**kw)
    s = lss.ImplicitHestonSolver(p)
    if adjoint_first:
        s.adjoint()
    s.line_chunks(17, 5)
    assert s.adjoint()[0] == s.solve()[1]
