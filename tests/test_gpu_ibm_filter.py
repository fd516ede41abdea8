"""IBM preprocessing with the FP32 filter ahead of the FP64 searches: bodies
near and far from the origin, triangles of all sizes and slivers, vertices
and edges through cell centres, open bodies whose cells fall back to the closest point.  Tables and flags equal
the oracle's restatement bit for bit."""
import numpy as np
import pytest

import oracle as O
from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _grid(shift=0.0, n=8):
    case = cases.sphere_cubes(64, n=n)
    case.origin = case.origin + shift
    return case


def _check(case, tris):
    fg, fo = case.fws.copy(), case.fws.copy()
    got = api.ibm_preprocess(case, tris, fg)
    want = O.Port().ibm(case, fo, tris)
    for x, y in zip(got, want):
        for a, b in zip(x, y):
            assert a.shape == b.shape
            assert np.array_equal(a.view(np.int64 if a.dtype == np.float64 else a.dtype),
                                  b.view(np.int64 if b.dtype == np.float64 else b.dtype))
    assert np.array_equal(fg, fo)
    return len(want[0][0]) + len(want[1][0])


@pytest.mark.parametrize("shift", [0.0, 3.0, 1.0e4])
@pytest.mark.parametrize("levels", [1, 3])
def test_bodies(shift, levels):
    tris = cases.icosphere(levels, 0.5, center=(0.004, -0.003, 0.002)) + shift
    _check(_grid(shift), tris)


@pytest.mark.parametrize("kind", ["open", "slivers", "on_cells", "one"])
def test_odd_triangles(kind):
    case = _grid()
    rng = np.random.RandomState(7)
    tris = cases.icosphere(3, 0.5, center=(0.004, -0.003, 0.002))
    if kind == "open":  # a third of the body missing
        tris = tris[rng.rand(len(tris)) < 0.67]
    elif kind == "slivers":  # from 1e-1 to 1e-9 of their height
        k = rng.randint(0, 10, len(tris))
        tris[:, 2] = tris[:, 0] + (tris[:, 2] - tris[:, 0]) * 10.0 ** -k[:, None]
    elif kind == "on_cells":  # vertices rounded to the cell centres' grid
        dx = case.cube_size[case.csl == 0][-1] / case.n
        tris = np.round(tris / dx - 0.5) * dx + 0.5 * dx
    else:
        tris = tris[:1]
    _check(case, np.ascontiguousarray(tris))
