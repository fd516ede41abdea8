"""FP64 LU-SGS sweeps by clusters of CTAs: every cluster size the launch
picks (by cube edge and cube count), planes of one cell and planes wider than
a CTA, rows that do not divide by the cluster, holes in the flow, and values
that take the fall-back from the integer division.  Bit-identical to the
oracle's serial sweep."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncx", [(4, 1), (8, 6), (12, 1), (16, 4), (20, 1), (24, 2), (24, 5),
                                   (28, 1), (32, 1)])
@pytest.mark.parametrize("tiny", [False, True])
def test_sweep_bitwise(n, ncx, tiny):
    case = cases.random_case(seed=n + ncx, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True,
                             solid_frac=0.03, ghost_frac=0.02, with_ibm=False)
    if tiny:
        r = cases.splitmix_uniform(3, case.U[..., 0].size).reshape(case.U.shape[:-1])
        case.U[r < 0.02, 1:4] = 0.0
        case.U[(r >= 0.02) & (r < 0.03), 2] *= 1e-310
    port = O.Port()
    port.set_threads(8)
    a = O.State(case)
    port.run_lusgs(case, a, 1, 2, 0.0, 1.5)
    ctx = api.CaseContext(case)
    ctx.set_method(api.METHOD_LUSGS)
    ctx.set_state(case.U, case.U, case.U)
    er = ctx.advance(1, 2)
    for x, y in zip((a.U1_, a.U1, a.U1q), ctx.get_state()):
        assert np.array_equal(x[1:], y[1:])
    # norms: sums of at most 1.7 M squares in another order
    assert np.allclose(er[1:6], a.er[1:6], rtol=1e-11, atol=0)
    ctx.close()
