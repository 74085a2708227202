"""The Polyakov loop's eight parts of the chain along t: fewer slices than parts, parts of unequal
length, slices of less than and not a whole number of 32 sites."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("link_reals", [12, 18])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 4, 6, 6), (4, 4, 4, 8), (6, 2, 4, 10),
                                  (4, 6, 10, 34), (8, 8, 8, 2)])
def test_polyakov(gfx, dims, link_reals):
    lx, ly, lz, lt = dims
    V = lx * ly * lz * lt
    u = gfx.random_init_haar(17, 4 * V)
    with gfx.Context(dims, link_reals=link_reals) as c:
        c.set_links(u)
        got = c.polyakov()
    m = (u[..., 0] + 1j * u[..., 1]).reshape(lt, lz * ly * lx, 4, 3, 3)[:, :, 3]
    p = m[0]
    for t in range(1, lt):
        p = p @ m[t]
    want = np.trace(p, axis1=1, axis2=2).mean() / 3.0
    # an entry of a product of unitary matrices is off by at most 6 roundings of sums below 2
    assert abs(got - want) < 2 * lt * 12 * 2.0 ** -53
