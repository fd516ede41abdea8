"""Convergence-driven stepping on the split path: eager and as a graph."""
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
