"""Split LU-SGS of many small cubes."""
import time

import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _us(case, method):
    ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    ctx.set_method(method)
    ctx.set_state(case.U, case.U, case.U)
    ctx.advance(1, 10)
    best = 1e9
    for _ in range(7):
        t = time.perf_counter()
        ctx.advance(2, 10)
        best = min(best, time.perf_counter() - t)
    ctx.close()
    return best / 20 * 1e6


@pytest.mark.parametrize("n,ncx,part", [(4, 16, 0.57), (8, 12, 0.64)])
def test_sub_iteration_of_many_small_cubes(n, ncx, part):
    """Against the three RK stages of the same cubes (one flux launch instead
    of three): CTAs of 256 threads for slabs of 16 and 64 cells and clusters of
    one CTA made it 0.65 and 0.70 of them, slower than one CTA a cube had been;
    now 0.52 and 0.60."""
    case = cases.taylor_green(ncx=ncx, n=n)
    assert _us(case, api.METHOD_LUSGS) < part * _us(case, api.METHOD_RK3)
