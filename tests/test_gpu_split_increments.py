"""What a sub-iteration of the split path adds to every cell, against the FP64
oracle's increment.

The bound.  A cell's increment is the balance of six face fluxes.  An FP32
flux holds some 60 roundings (2^-24) of its terms; with fields of 5% noise the
largest term, the mean flow's convective flux, is some 20 times the flux
differences that make the increment: 6 x 60 x 20 / 2^24 = 4e-4 of the largest
increment, twice that with the preconditioner's and the three stages' own.
Another reconstruction order at one face changes its flux by a part of the
noise itself, a tenth of an increment and more (checked on the CPU below)."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

BOUND = 1e-3


def _case(n, ncx, viscous=True, seed=None):
    return cases.random_case(seed=n if seed is None else seed, n=n, ncx=ncx, ncy=ncx, ncz=ncx,
                             periodic=True, viscous=viscous, with_ibm=False)


def _interior(a):
    return a[1:, 2:-2, 2:-2, 2:-2]


def _oracle_increment(case, port=None):
    port = port or O.Port()
    port.set_threads(8)
    st = O.State(case)
    port.run(case, st, 1, 1)
    return _interior(st.U1_ - case.U)


def _errors(x, ref):
    """Per variable the largest error of any cell and the L2 error, both of
    the oracle's increment's."""
    d = np.abs(x - ref)
    return (d.max(axis=(0, 1, 2, 3)) / np.abs(ref).max(axis=(0, 1, 2, 3)),
            np.sqrt((d ** 2).sum(axis=(0, 1, 2, 3)) / (ref ** 2).sum(axis=(0, 1, 2, 3))))


# (n, cubes an axis): 4^3 tiles, one 8^3 tile a cube (729 cubes), the march by
# compile-time and run-time sizes, edges of several 8^3 tiles
@pytest.mark.gpu
@pytest.mark.parametrize("n,ncx", [(4, 3), (8, 2), (8, 9), (12, 2), (16, 2), (16, 4), (20, 2),
                                   (24, 2), (28, 1), (32, 1), (36, 1), (40, 1), (44, 1), (56, 1),
                                   (88, 1)])
@pytest.mark.parametrize("viscous", [True, False])
@pytest.mark.parametrize("form", [0, 2])
def test_increment_of_every_cell(n, ncx, viscous, form):
    case = _case(n, ncx, viscous)
    ref = _oracle_increment(case)
    ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    ctx.set_tuning(flux_form=form)
    ctx.set_state(case.U, case.U, case.U)
    ctx.advance(1, 1)
    x = _interior(ctx.get_state()[0] - case.U)
    ctx.close()
    cell, norm = _errors(x, ref)
    assert cell.max() < BOUND and norm.max() < BOUND, (cell, norm)
    assert not x[_interior(case.fws) != cases.IFLUID].any()


def test_the_bound_sees_a_missing_update_and_one_wrong_face():
    """Planted in the oracle: no update at all, and one solid cell flagged
    fluid, which gives the faces around it other reconstruction orders (its
    neighbours' increments are compared, not its own; solid cells with fluid
    ones on both sides along an axis, away from the cube's faces: elsewhere
    the orders are low already)."""
    case = _case(16, 1)
    ref = _oracle_increment(case)
    cell, norm = _errors(np.zeros_like(ref), ref)
    assert cell.min() >= 1 and norm.min() >= 1
    fluid = _interior(case.fws) == cases.IFLUID
    planted = 0
    for c, i, j, k in np.argwhere(~fluid):
        if not (3 <= i < 13 and fluid[c, i - 3:i, j, k].all() and fluid[c, i + 1:i + 4, j, k].all()):
            continue
        wrong = _case(16, 1)
        wrong.fws[c + 1, i + 2, j + 2, k + 2] = cases.IFLUID
        x = _oracle_increment(wrong)
        x[c, i, j, k] = ref[c, i, j, k]
        cell, _ = _errors(x, ref)
        assert cell.max() > 10 * BOUND, ((c, i, j, k), cell)
        planted += 1
        if planted == 8:
            break
    assert planted == 8
