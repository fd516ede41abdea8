"""Device memory of the split path: LU-SGS sweeps and the flux twin need no
more than the arrays a context holds anyway."""
import numpy as np
import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu

GRAIN = 4 << 20  # what the driver may take beside the arrays (2 MiB pages)


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("n,ncx", [(8, 12), (32, 4)])
def test_lusgs_takes_no_memory_of_its_own(n, ncx):
    case = cases.taylor_green(ncx=ncx, n=n)
    ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    ctx.set_state(case.U, case.U, case.U)
    ctx.advance(1, 1)
    before = _used()
    ctx.set_method(api.METHOD_LUSGS)
    ctx.advance(1, 1, use_graph=False)
    # 4 bytes a cell would be 3.5 and 8.4 MB: both sides of the grain
    assert _used() - before <= GRAIN + 4 * case.n_cells
    ctx.close()


@pytest.mark.parametrize("n", [4, 32])
def test_scratch_and_codes_keep_apart(n):
    """RK steps after LU-SGS ones (the cell codes lie beside the sweep's
    scratch) give the bits of a context that never ran LU-SGS."""
    case = cases.random_case(seed=n, n=n, ncx=1, ncy=1, ncz=2, periodic=True, with_ibm=False)
    out = []
    for lusgs_first in (True, False):
        ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
        if lusgs_first:
            ctx.set_state(case.U, case.U, case.U)
            ctx.set_method(api.METHOD_LUSGS)
            ctx.advance(1, 2)
            ctx.set_method(api.METHOD_RK3)
        ctx.set_state(case.U, case.U, case.U)
        ctx.advance(1, 2)
        out.append(ctx.get_state())
        ctx.close()
    for x, y in zip(*out):
        assert np.array_equal(x[1:].view(np.uint64), y[1:].view(np.uint64))
