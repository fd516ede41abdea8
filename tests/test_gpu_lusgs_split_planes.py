"""Split LU-SGS sweeps: one CTA per cube and clusters of four, planes of one
cell and planes wider than the CTA, rows that do not divide by the cluster,
holes in the flow and a single pass or several over a plane."""
import numpy as np
import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _increment(case, prec, threads=0):
    ctx = api.CaseContext(case, prec)
    ctx.set_method(api.METHOD_LUSGS)
    if threads:
        ctx.set_tuning(lusgs_threads=threads)
    ctx.set_state(case.U, case.U, case.U)
    er = ctx.advance(1, 1)
    U = ctx.get_state()[0]
    ctx.close()
    return er, U, (U - case.U)[1:, 2:-2, 2:-2, 2:-2]


@pytest.mark.parametrize("n,ncx", [(4, 1), (8, 3), (12, 2), (20, 1), (24, 2), (16, 3), (28, 1),
                                   (32, 1), (32, 5)])
def test_split_sweep(n, ncx):
    """Every cell's increment of a sub-iteration against the FP64 sweep.  The
    diagonal dominates (the sweep damps what it carries), so a cell holds some
    hundred FP32 roundings (2^-24) of terms no larger than the largest
    increment: 1e-3 of that leaves a factor of 100, while a wrong neighbour or
    row shows as 0.1 or more.  Passes of one warp over the planes change no
    bit."""
    case = cases.random_case(seed=n + ncx, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True,
                             solid_frac=0.03, ghost_frac=0.02, with_ibm=False)
    _, _, ref = _increment(case, api.PRECISION_FP64)
    er, U, x = _increment(case, api.PRECISION_SPLIT)
    scale = np.abs(ref).max(axis=(0, 1, 2, 3))
    assert (np.abs(x - ref).max(axis=(0, 1, 2, 3)) / scale).max() < 1e-3
    er1, U1, _ = _increment(case, api.PRECISION_SPLIT, 32)
    assert np.array_equal(U[1:].view(np.uint64), U1[1:].view(np.uint64))
    assert np.array_equal(er, er1)
