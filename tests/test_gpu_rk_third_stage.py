"""FP64 third RK stage: values that take the fall-back from the integer
products and divisions (zeros, subnormal and tiny momenta, tiny states) beside
ordinary ones.  States equal the oracle's bit for bit; norms are sums in
another order."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncx", [(4, 1), (4, 3), (12, 2)])
@pytest.mark.parametrize("tiny", [False, True])
def test_third_stage_bitwise(n, ncx, tiny):
    case = cases.random_case(seed=n + ncx, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True,
                             with_ibm=False)
    if tiny:
        r = cases.splitmix_uniform(3, case.U[..., 0].size).reshape(case.U.shape[:-1])
        case.U[r < 0.02, 1:4] = 0.0
        case.U[(r >= 0.02) & (r < 0.04), 2] *= 1e-310
    port = O.Port()
    a = O.State(case)
    port.run(case, a, 1, 1)
    ctx = api.CaseContext(case)
    ctx.set_state(case.U, case.U, case.U)
    er = ctx.advance(1, 1)
    for x, y in zip((a.U1_, a.U1, a.U1q), ctx.get_state()):
        assert np.array_equal(x[1:], y[1:])
    assert np.allclose(er[1:6], a.er[1:6], rtol=1e-11, atol=0)
    assert np.allclose(ctx.emax[1:6], a.Emax[1:6], rtol=1e-11, atol=0)
    ctx.close()
