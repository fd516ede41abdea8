"""A step that stops on an error of its exchange hook leaves nothing behind
that a later call would run."""
import numpy as np
import pytest

from bcm_cgli_gb300 import _lib, api, cases
from bcm_cgli_gb300._lib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_SPLIT])
@pytest.mark.parametrize("method", [api.METHOD_RK3, api.METHOD_LUSGS])
@pytest.mark.parametrize("fail_at", [1, 2])  # the opening, the closing interface call
def test_timing_after_a_failed_exchange_keeps_the_state(precision, method, fail_at):
    case = cases.random_case(seed=4, n=8, periodic=True, with_ibm=False)
    ctx = api.CaseContext(case, precision=precision)
    ctx.set_method(method)
    ctx.set_state(case.U, case.U, case.U)
    calls = []

    def hook(user, phase, stream):
        if phase == api.XCHG_HALO:
            calls.append(phase)
            return len(calls) == fail_at
        return 0

    fn = _lib.EXCHANGE_FN(hook)
    api.check(lib().bcmg_case_set_exchange(ctx.h, fn, None))
    with pytest.raises(api.BcmgError):
        ctx.advance(1, 1, use_graph=False)
    api.check(lib().bcmg_case_set_exchange(ctx.h, _lib.EXCHANGE_FN(), None))
    before = ctx.get_state()
    ctx.time_flux(1)
    for x, y in zip(before, ctx.get_state()):
        assert np.array_equal(x[1:].view(np.uint64), y[1:].view(np.uint64))
    ctx.close()
