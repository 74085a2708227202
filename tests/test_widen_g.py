"""FP32 g widened to FP64: rows 0, 1 of a single-precision field orthonormalized to FP64 accuracy,
for rows near unitary (fixed point) and far from it (FP64), against Gram-Schmidt in extended
precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the rows' deviation from unitary: rounding only, below and above the fixed-point bound, scaled
@pytest.mark.parametrize("noise,scale", [(0.0, 1.0), (1e-4, 1.0), (1e-2, 1.0), (0.0, 1.5)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 6, 2, 10)])
def test_widened_rows(gfx, dims, noise, scale):
    V = int(np.prod(dims))
    g = gfx.random_init_haar(23, V)
    rng = np.random.RandomState(1)
    g = scale * (g + noise * rng.standard_normal(g.shape))
    g[0] = scale * np.eye(3)[:, :, None] * np.array([1.0, 0.0])
    with gfx.Context(dims, precision=gfx.PREC_MIXED) as c:
        c.set_links(gfx.random_init_haar(3, 4 * V))
        c.set_trafo(g)
        c.functional(gfx.LANDAU, 0)  # makes the FP32 copy the current g
        got = c.get_trafo()
    r = g.astype(np.float32).astype(np.longdouble)
    z = r[..., 0] + 1j * r[..., 1]
    a, b = z[:, 0], z[:, 1]
    a = a / np.sqrt((abs(a) ** 2).sum(1, keepdims=True))
    b = b - (b * a.conj()).sum(1, keepdims=True) * a
    b = b / np.sqrt((abs(b) ** 2).sum(1, keepdims=True))
    want = np.stack([a, b], 1)
    # entries below 1; a dozen roundings each in FP64, half an ulp in fixed point
    d = got[:, :2, :, 0] + 1j * got[:, :2, :, 1] - want
    assert abs(d).max() < 12 * 2.0 ** -53
