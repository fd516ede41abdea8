"""The autotuner: the shape a context runs by default is timed at every edge,
and LU-SGS sweeps of different widths on the context's own residual."""
import numpy as np
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


def _tuned(case, reps):
    ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    ctx.set_method(api.METHOD_LUSGS)
    ctx.set_state(case.U, case.U, case.U)
    res = ctx.autotune(reps)
    increments = ctx.get_scratch()[2]  # split path: the last sweep's increment among them
    ctx.close()
    return res, increments


@pytest.mark.parametrize("n", [16, 32])
def test_sweeps_are_timed_on_the_residual(n):
    """The last timed sweep solves the context's own residual, however many
    came before it (a sweep leaves its increment in the residual's place)."""
    case = cases.random_case(seed=n, n=n, ncx=1, ncy=1, ncz=1, periodic=True, with_ibm=False)
    one, three = _tuned(case, 1), _tuned(case, 3)
    assert np.array_equal(one[1].view(np.uint64), three[1].view(np.uint64))


@pytest.mark.parametrize("n,half", [(28, 96), (32, 96)])
def test_sweep_candidates_differ_where_four_ctas_sweep_a_cube(n, half):
    """A CTA's widest plane has 147 (28) and 192 cells (32): half of it is 96
    threads.  Half of the cube's widest plane (320, 384) ran the same launch."""
    case = cases.taylor_green(ncx=4, n=n)
    for _ in range(4):
        res, _ = _tuned(case, 2)
        assert res["lusgs_threads"] in (0, half)
        # two passes over every wide plane: never free
        assert res["lusgs_ms"]["half"] > 1.03 * res["lusgs_ms"]["widest"]
