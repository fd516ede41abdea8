"""Contexts of different cube edges stepped by threads side by side: the launch
limits a kernel is given do not depend on whose launch comes between."""
import threading

import pytest

from bcm_cgli_gb300 import api, cases

pytestmark = pytest.mark.gpu


def _beside(make, work):
    """Runs work(context) in a thread per context, all at once."""
    ctxs = [make(i) for i in range(2)]
    errs, gate = [], threading.Barrier(len(ctxs))

    def run(ctx):
        try:
            gate.wait()
            work(ctx)
        except Exception as exc:
            errs.append(exc)

    ts = [threading.Thread(target=run, args=(c,)) for c in ctxs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for c in ctxs:
        c.close()
    assert not errs, errs[0]


@pytest.mark.parametrize("edges,precision,lusgs", [
    ((12, 20), api.PRECISION_FP64, False),  # boxes of different sizes
    ((36, 44), api.PRECISION_SPLIT, False),  # the march's run-time sizes
    ((8, 24), api.PRECISION_FP64, True),
    ((8, 24), api.PRECISION_SPLIT, True),  # planes of different widths
])
def test_two_edges_side_by_side(edges, precision, lusgs):
    def make(i):
        case = cases.random_case(seed=i, n=edges[i], ncx=1, ncy=1, ncz=1, periodic=True,
                                 with_ibm=False)
        ctx = api.CaseContext(case, precision=precision)
        if lusgs:
            ctx.set_method(api.METHOD_LUSGS)
        ctx.set_state(case.U, case.U, case.U)
        return ctx

    def work(ctx):
        for _ in range(10):
            if lusgs:
                ctx.advance(1, 100, use_graph=False)
            else:
                ctx.time_flux(1000)

    _beside(make, work)
