"""Norms of 8^3 cubes with one face per thread and turn (flux_form 2): the
march (few cubes) and the tiles (700 and more) sum in one order."""
import numpy as np
import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _wide_range(seed):
    """Perturbations that fall by a decade per cell along k, so that the squares
    of a row, which a warp sums, span some 14 decades and any other order of
    the sums rounds differently."""
    case = cases.random_case(seed=seed, n=8, periodic=True, with_ibm=False, solid_frac=0.0,
                             ghost_frac=0.0)
    ph = case.phys
    r = [cases.splitmix_uniform(seed + t, case.U[..., 0].size).reshape(case.U.shape[:-1]) - 0.5
         for t in range(5)]
    a = 10.0 ** -np.abs(np.arange(case.S, dtype=float) - 2)
    case.U = np.ascontiguousarray(cases.conservative(
        ph.rho0 * (1 + 0.05 * a * r[0]), ph.U0 * a * r[1], ph.U0 * a * r[2], ph.U0 * a * r[3],
        ph.P0 * (1 + 0.01 * a * r[4])))
    return case


@pytest.mark.parametrize("form", [0, 2])
def test_norms_alone_and_in_a_large_batch(form):
    big = cases.random_case(seed=8, n=8, ncx=9, ncy=9, ncz=9, periodic=True, with_ibm=False)
    small = [_wide_range(s) for s in (11, 23, 37)]
    b = api.BatchContext(small + [big], precision=api.PRECISION_SPLIT)
    b.set_tuning(flux_form=form)
    for q, c in enumerate(small + [big]):
        b.set_case_state(q, c.U, c.U, c.U)
    er = b.advance(1, 1)
    for q, c in enumerate(small):
        a = api.CaseContext(c, precision=api.PRECISION_SPLIT)
        a.set_tuning(flux_form=form)
        a.set_state(c.U, c.U, c.U)
        e = a.advance(1, 1)
        assert np.array_equal(a.get_state()[0][1:], b.get_case_state(q)[0][1:])
        assert np.array_equal(e[1:], er[q, 1:])
        assert np.array_equal(np.ravel(a.emax)[1:6], np.ravel(b.emax)[6 * q + 1:6 * q + 6])
        a.close()
    b.close()
