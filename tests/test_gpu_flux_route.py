"""The split stage's kernel by cube edge: an edge divisible by 8 costs no more
per cell than the 8^3 tiles do at an edge only they serve."""
import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _ns_per_cell(n, ncx):
    case = cases.taylor_green(ncx=ncx, n=n)
    ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    ctx.set_state(case.U, case.U, case.U)
    ctx.time_flux(3)
    ms = min(ctx.time_flux(10) for _ in range(5))
    ctx.close()
    return 1e6 * ms / case.n_cells


def test_large_edges_cost_what_the_tiles_cost():
    """3 to 5 million cells each (many waves of CTAs).  The wrong kernel took
    1.24 (56), 1.73 (72) and 1.56 (80) times the tiles' time per cell; the
    edges' own differ by 4% (waves, ghost layers)."""
    tiles = _ns_per_cell(88, 2)
    for n, ncx in ((40, 4), (48, 3), (56, 3), (72, 2), (80, 2)):
        assert _ns_per_cell(n, ncx) < 1.12 * tiles, n
