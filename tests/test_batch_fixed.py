"""Batched copies have the bits of their single-lattice solves wherever FP64-accurate sweeps run:
DOUBLE batches, MIXED ones polished in FP64, links and starts that keep to the FP64 kernels."""
import numpy as np
import pytest

from conftest import haar, smooth_links

pytestmark = pytest.mark.gpu

CONFS = [((4, 4, 6, 8), 3), ((8, 8, 8, 12), 2), ((4, 6, 4, 10), 2)]


def _inputs(double):
    links, starts = [], []
    for k, (dims, n) in enumerate(CONFS):
        u = smooth_links(dims, 0.35, 90 + k)
        if k == 2 and double:
            # further from unitary than the fixed-point arithmetic takes (FP32 sweeps, whose
            # reduced forms are for unitary links, do not converge on them)
            u *= 1.01
        links.append(u)
        gs = [haar(int(np.prod(dims)), 100 + 10 * k + c) for c in range(n)]
        if k < 2:  # read from 32-bit data: the first sweep is an FP64 one
            gs[1] = gs[1].astype(np.float32).astype(np.float64)
        starts.append(gs)
    return links, starts


@pytest.mark.parametrize("use_graph", [1, 0])
@pytest.mark.parametrize("gauge", [0, 1])
@pytest.mark.parametrize("precision,polish", [("PREC_DOUBLE", 0), ("PREC_MIXED", 0),
                                              ("PREC_MIXED", 2)])
def test_copies_are_single_solves(gfx, precision, polish, gauge, use_graph):
    precision = getattr(gfx, precision)
    links, starts = _inputs(precision == gfx.PREC_DOUBLE)
    p = gfx.Context.or_params(maxit=20000, eps=1e-13, checkinterval=15, omega=1.7, gauge=gauge,
                              criterion=gfx.CRIT_THETA, checkinterval_double=3, polish=polish,
                              use_graph=use_graph)
    b = gfx.Batch([d for d, _ in CONFS], [n for _, n in CONFS], precision=precision)
    for k in range(len(CONFS)):
        b.set_links(k, links[k])
    for again in range(2):  # the second solve has the fields and graphs of the first
        for k, gs in enumerate(starts):
            for c, g in enumerate(gs):
                b.set_trafo(k, c, g)
        res, _ = b.overrelax(p)
    at = 0
    for k, (dims, n) in enumerate(CONFS):
        s = gfx.Context(dims, precision=precision)
        s.set_links(links[k])
        for c in range(n):
            s.set_trafo(starts[k][c])
            r = s.overrelax(p)
            assert r.converged and res[at]["converged"]
            assert res[at]["iterations"] == r.iterations
            assert res[at]["F"] == r.final_values.F
            assert np.array_equal(b.get_trafo(k, c), s.get_trafo()), (k, c)
            at += 1
        s.close()
    b.close()
