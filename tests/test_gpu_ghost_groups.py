"""IBM ghost fill by groups of entries: components of cubes with all their
levels in one launch, and tables that link or crowd the cubes and run a level
per launch; ghosts inside their own stencil (with weights next to 1), values
that take the fall-back from the integer divisions, tables of one entry and of
one more than a CTA's pass.  Bit-identical to the oracle's serial loop."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _fill(case, tables, tiny):
    api.reference_config_for(case)
    U = case.U.copy()
    if tiny:
        r = cases.splitmix_uniform(5, U[..., 0].size).reshape(U.shape[:-1])
        U[r < 0.03, 1:4] = 0.0
        U[(r >= 0.03) & (r < 0.06), 2] *= 1e-310
        U[(r >= 0.06) & (r < 0.08)] *= 1e-200
    port = O.Port()
    for which, t in zip((-1, 1), tables):
        W, G, I = t
        case.ibm_minus, case.ibm_plus = (t, None) if which < 0 else (None, t)
        a, b = U.copy(), U.copy()
        port.ghost(case, a, which)
        f = api.BCM_Ghostcell_minus if which < 0 else api.BCM_Ghostcell_plus
        f(0, (len(G) - 1) // 4, W, G, I, case.fws, b)
        assert np.array_equal(a, b)


def _cut(t, m):
    W, G, I = t
    return (np.ascontiguousarray(W[:8 * m + 1]), np.ascontiguousarray(G[:4 * m + 1]),
            np.ascontiguousarray(I[:4 * m + 1]))


@pytest.mark.parametrize("tiny", [False, True])
@pytest.mark.parametrize("entries", [1, 32, 33, None])
def test_sphere_groups(entries, tiny):
    case = cases.sphere_cubes(64, n=8, mach=0.2, reynolds=150.0, seed=11)
    t = case.ibm_minus
    if entries:
        t = _cut(t, entries)
    _fill(case, (t, t), tiny)


@pytest.mark.parametrize("tiny", [False, True])
@pytest.mark.parametrize("n,ncx,cross", [(4, 2, False), (4, 2, True), (16, 1, False), (8, 2, True)])
def test_random_tables(n, ncx, cross, tiny):
    """Random entries: up to some hundred levels in a cube, every entry's stencil
    in its ghost's cube or (cross) in any."""
    case = cases.random_case(seed=n, n=n, ncx=ncx, ncy=ncx, ncz=ncx, with_ibm=False)
    m, rng = 60 * n, np.random.RandomState(n + cross)
    G, I, W = np.zeros((m, 4), np.int32), np.zeros((m, 4), np.int32), rng.rand(m, 8)
    G[:, 0] = rng.randint(1, case.ncube, m)
    I[:, 0] = rng.randint(1, case.ncube, m) if cross else G[:, 0]
    I[:, 1:] = rng.randint(1, n + 2, (m, 3))
    near = rng.rand(m) < 0.5  # ghost inside its stencil
    G[:, 1:] = np.where(near[:, None], I[:, 1:] + rng.randint(0, 2, (m, 3)),
                        rng.randint(0, n + 4, (m, 3)))
    W /= W.sum(1, keepdims=True)
    W[::7] = 0.0
    W[::7, rng.randint(0, 8)] = 1.0
    one = lambda x, dt: np.concatenate([np.zeros(1, dt), x.ravel().astype(dt)])
    t = (one(W, np.float64), one(G, np.int32), one(I, np.int32))
    _fill(case, (t, t), tiny)
