"""Ghost layers of a stage in one launch: closing interface call, boundary
conditions and opening call of a cube by a cluster of CTAs, for every cluster
size the launch picks (by cube count and edge), boundary faces that a periodic
neighbour also fills, open boxes, level jumps and IBM ghost cells (whose fill
lies between the passes).  Every cell, ghost layers included, equals the
oracle's serial calls bit for bit."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _case(kind, n, ncx, periodic):
    if kind == "levels":
        return cases.random_two_level_case(seed=n + ncx, n=n, ncx=ncx, ncy=ncx, ncz=ncx,
                                           periodic=periodic)
    return cases.random_case(seed=n + ncx, n=n, ncx=ncx, ncy=ncx, ncz=ncx, periodic=periodic,
                             with_ibm=kind == "ibm")


@pytest.mark.parametrize("kind,n,ncx", [("plain", 4, 1), ("plain", 4, 5), ("plain", 4, 7),
                                        ("plain", 16, 2), ("plain", 16, 5), ("ibm", 4, 5),
                                        ("ibm", 8, 2), ("levels", 4, 2), ("levels", 4, 5),
                                        ("levels", 12, 2)])
@pytest.mark.parametrize("periodic", [False, True])
def test_stage_layers_bitwise(kind, n, ncx, periodic):
    case = _case(kind, n, ncx, periodic)
    port = O.Port()
    port.set_threads(8)
    a = O.State(case)
    port.run(case, a, 2, 2)
    for graph in (False, True):
        ctx = api.CaseContext(case)
        ctx.set_state(case.U, case.U, case.U)
        er = ctx.advance(2, 2, use_graph=graph)
        for x, y in zip((a.U1_, a.U1, a.U1q), ctx.get_state()):
            assert np.array_equal(x[1:], y[1:])
        assert np.allclose(er[1:6], a.er[1:6], rtol=1e-11, atol=0)
        ctx.close()
