"""What a context keeps between calls: the results of a call do not depend on which calls came
before it."""
import numpy as np
import pytest

from conftest import haar, smooth_links

pytestmark = pytest.mark.gpu


def _context(gfx, dims, u, g, **kw):
    c = gfx.Context(dims, **kw)
    c.set_links(u)
    c.set_trafo(g)
    return c


@pytest.mark.parametrize("precision", ["PREC_DOUBLE", "PREC_MIXED"])
def test_history_of_a_longer_solve(gfx, precision):
    # the same loop (interval, omega) with room for more checks than the first solve had
    dims = (4, 4, 6, 8)
    u, g = smooth_links(dims, 0.4, 31), haar(int(np.prod(dims)), 32)
    kw = dict(eps=1e-12, checkinterval=1, omega=1.7, criterion=gfx.CRIT_THETA)
    a, b = (_context(gfx, dims, u, g, precision=getattr(gfx, precision)) for _ in range(2))
    a.overrelax(maxit=5, **kw)
    a.set_trafo(g)
    ra, rb = (c.overrelax(maxit=5000, **kw) for c in (a, b))
    assert ra.iterations == rb.iterations > 0
    assert len(a.history()) > 10 and a.history() == b.history()
    assert np.array_equal(a.get_trafo(), b.get_trafo())
    a.close()
    b.close()
