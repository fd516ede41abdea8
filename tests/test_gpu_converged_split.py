"""Convergence-driven stepping: eager and as a graph on the split path, and
after a change of the LU-SGS parameters."""
import numpy as np
import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [api.METHOD_RK3, api.METHOD_LUSGS])
def test_eager_steps_equal_graph_steps(method):
    """The first step after a state was set, and a batch whose cases stop at
    different sub-iterations (a case that sat some out is mirrored again)."""
    cs = [cases.taylor_green(ncx=2, n=8), cases.random_case(seed=3, n=8, periodic=True),
          cases.random_two_level_case(seed=6, n=8, periodic=False)]
    out = []
    for graph in (True, False):
        b = api.BatchContext(cs, precision=api.PRECISION_SPLIT)
        b.set_method(method)
        for q, c in enumerate(cs):
            b.set_case_state(q, c.U, c.U, c.U)
        er, its = b.advance_converged(2, 30, 0.05, use_graph=graph)
        out.append([er, its] + list(b.get_state()))
        b.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_SPLIT])
def test_new_lusgs_parameters_reach_the_captured_step(precision):
    case = cases.taylor_green(ncx=2, n=8)
    out = []
    for before in (True, False):
        ctx = api.CaseContext(case, precision=precision)
        if before:  # a step graph with other parameters
            ctx.set_method(api.METHOD_LUSGS, cfl=0.0, omega=1.5)
            ctx.set_state(case.U, case.U, case.U)
            ctx.advance_converged(1, 4, 1e-3)
        ctx.set_method(api.METHOD_LUSGS, cfl=2.0, omega=1.1)
        ctx.set_state(case.U, case.U, case.U)
        ctx.emax[:] = 0
        ctx.advance_converged(1, 4, 1e-3)
        out.append(ctx.get_state()[0])
        ctx.close()
    assert np.array_equal(*out)
