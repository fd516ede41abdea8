"""The split-precision stage's march along i (bcm_flux_march.cu): cube edges
with compile-time and run-time sizes, one tile and several per cross-section,
march segments that start inside a cube, holes in the flow (second views of
faces inside tiles, at tile ends and at segment ends), against the FP64
oracle; and independence of how many cubes share a launch."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncx", [(8, 2), (12, 2), (16, 2), (16, 4), (20, 2), (24, 2), (28, 1),
                                   (32, 1), (36, 1), (40, 1)])
@pytest.mark.parametrize("viscous", [True, False])
@pytest.mark.parametrize("form", [0, 2])
def test_stages_against_oracle(n, ncx, viscous, form):
    case = cases.random_case(seed=n, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True,
                             viscous=viscous, with_ibm=False)
    port = O.Port()
    port.set_threads(8)
    a = O.State(case)
    port.run(case, a, 1, 2)
    ctx = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    ctx.set_tuning(flux_form=form)
    ctx.set_state(case.U, case.U, case.U)
    er = ctx.advance(1, 2)
    U1_ = ctx.get_state()[0]
    # every variable's change over the step within 1e-5 relative L2 (the split
    # path's stated bound), ghost cells included
    for v in range(5):
        d = np.linalg.norm(U1_[1:, ..., v] - a.U1_[1:, ..., v])
        scale = np.linalg.norm(a.U1_[1:, ..., v]) if v in (0, 4) else np.linalg.norm(
            a.U1_[1:, ..., 1:4])
        assert d <= 1e-5 * scale, (v, d / scale)
    # norms: FP32 increments of a noisy field (5% perturbation, condition
    # number of the residual differences about 1e3 x 6e-8)
    assert np.allclose(er[1:6], a.er[1:6], rtol=1e-3)
    assert np.array_equal(ctx.mirror_current()[1:], ctx.mirror()[1:])
    ctx.close()


@pytest.mark.parametrize("n,ncx", [(8, 9), (16, 3)])
def test_same_bits_however_the_cubes_are_launched(n, ncx):
    """A context of all cubes against two ranks with half of them each (other
    segments per CTA; for n = 8 the tile kernel against the march)."""
    case = cases.random_case(seed=5, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=True, with_ibm=False)
    one = api.CaseContext(case, precision=api.PRECISION_SPLIT)
    one.set_state(case.U, case.U, case.U)
    one.advance(1, 2, use_graph=False)
    ranks = np.zeros(case.ncube, np.int32)
    ranks[1 + (case.ncube - 1) // 2:] = 1
    two = api.ShardedRun(case, ranks, precision=api.PRECISION_SPLIT)
    two.set_state(case.U, case.U, case.U)
    two.advance(1, 2)
    s = (slice(1, None),) + (slice(2, -2),) * 3
    assert np.array_equal(one.get_state()[0][s], two.get_state()[0][s])
    two.close()
    one.close()


def test_norms_of_a_case_do_not_depend_on_its_batch():
    """n = 8: a small case alone (march) and in a batch of over 700 cubes
    (tiles) gets the same norms, bit for bit."""
    small = cases.random_case(seed=7, n=8, periodic=True)
    big = cases.random_case(seed=8, n=8, ncx=9, ncy=9, ncz=9, periodic=True)
    alone = api.CaseContext(small, precision=api.PRECISION_SPLIT)
    alone.set_state(small.U, small.U, small.U)
    e0 = alone.advance(1, 2)
    b = api.BatchContext([small, big], precision=api.PRECISION_SPLIT)
    for q, c in enumerate((small, big)):
        b.set_case_state(q, c.U, c.U, c.U)
    e1 = b.advance(1, 2)
    assert np.array_equal(alone.get_state()[0][1:], b.get_case_state(0)[0][1:])
    assert np.array_equal(e0[1:], e1[0, 1:])
    b.close()
    alone.close()
