"""Neighbour lists of a case (interface_lists) for every integer type of the
level array: unsigned levels have no negative differences."""
import numpy as np
import pytest

from bcm_cgli_gb300 import api, cases


def _lists(case):
    """The lists cube by cube, from the comparisons that define them."""
    out = []
    for ax in range(3):
        eq, bsp, sbp, bsm, sbm = [], [], [], [], []
        for c in range(1, case.ncube):
            a, b = (int(case.adj[c, 1:5, s + 2 * ax].max()) for s in (2, 1))
            if a > 0:
                (eq if case.csl[c] == case.csl[a] else sbp if case.csl[c] < case.csl[a]
                 else bsp).append(c)
            if b > 0 and case.csl[c] != case.csl[b]:
                (sbm if case.csl[c] < case.csl[b] else bsm).append(c)
        out.append([eq, bsp, sbp, bsm, sbm])
    return out


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.uint8, np.uint32, np.uint64])
def test_lists_by_level_type(dtype):
    case = cases.random_two_level_case(seed=5, n=4, ncx=3, ncy=2, ncz=2)
    want = _lists(case)
    assert all(any(want[ax][k] for ax in range(3)) for k in range(5))
    case.csl = case.csl.astype(dtype)
    for w, got in zip(want, api.interface_lists(case)):
        assert [list(g[1:]) for g in got] == w
