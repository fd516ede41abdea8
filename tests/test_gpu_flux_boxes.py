"""FP64 flux boxes of cube edges that 8 does not divide: one box a CTA and
several, a last CTA that is not full, boxes of one wave and of many, whole and
thin ones, with solids (the boxes of a CTA share its second views)."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncx", [(4, 1), (4, 3), (4, 5), (4, 6), (4, 11), (12, 1), (12, 2),
                                   (12, 3), (12, 4), (12, 5), (20, 1), (20, 2), (28, 1), (36, 1),
                                   (44, 1), (52, 1)])
@pytest.mark.parametrize("viscous", [True, False])
def test_stage_bits(n, ncx, viscous):
    case = cases.random_case(seed=n + ncx, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True,
                             viscous=viscous, solid_frac=0.05, ghost_frac=0.03, with_ibm=False)
    port = O.Port()
    port.set_threads(8)
    a = O.State(case)
    port.run(case, a, 1, 1)
    ctx = api.CaseContext(case)
    ctx.set_state(case.U, case.U, case.U)
    ctx.advance(1, 1)
    assert np.array_equal(ctx.get_state()[0][1:].view(np.uint64), a.U1_[1:].view(np.uint64))
    ctx.close()


def test_few_cubes_spread_over_the_chip():
    """Few cubes fill no wave with large CTAs, so they take small ones: a
    launch over them is a small part of one over many (with CTAs of 400 to
    500 cells whatever the number of cubes it was 0.34, 0.50 and 0.25)."""
    def ms(n, ncx):
        case = cases.random_case(seed=1, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True,
                                 with_ibm=False)
        ctx = api.CaseContext(case)
        ctx.set_state(case.U, case.U, case.U)
        ctx.time_flux(2)
        t = min(ctx.time_flux(5) for _ in range(3))
        ctx.close()
        return t

    for n, few, many, part in ((20, 1, 3, 0.22), (12, 1, 4, 0.33), (4, 2, 16, 0.16)):
        assert ms(n, few) < part * ms(n, many), n
