"""The autotuner times the shape a context runs by default, at every edge."""
import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncx", [(12, 6), (20, 4)])
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_SPLIT])
def test_default_shape_is_a_candidate_where_8_does_not_divide(n, ncx, precision):
    """At these sizes the default (the march, large boxes) is well ahead of the
    4^3 tiles: 2.4 times on the split path, 1.15 in FP64."""
    case = cases.taylor_green(ncx=ncx, n=n)
    ctx = api.CaseContext(case, precision=precision)
    ctx.set_state(case.U, case.U, case.U)
    ctx.time_flux(2)
    default = min(ctx.time_flux(5) for _ in range(3))
    res = ctx.autotune(5)
    assert res["flux_ms"]["8_packed"] > 0 and res["flux_ms"]["4"] > 0
    assert res["flux_tile"] == 0
    assert min(ctx.time_flux(5) for _ in range(3)) < 1.1 * default
    ctx.close()
