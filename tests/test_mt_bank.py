"""The twister bank's kernel at the edges of its steps (ten outputs of a twister), tiles (160)
and ring (19): bit-exact uniforms, states and seeds against the oracle over several updates."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# outputs per twister (made even): the smallest; below, at and beyond a step, the ring, a tile
@pytest.mark.parametrize("per_g,per_u", [(2, 2), (10, 8), (12, 20), (18, 38), (20, 158),
                                         (160, 162), (190, 320), (330, 182)])
def test_uniforms_states_and_seeds(gfx, oracle, mt_params, per_g, per_u):
    c = gfx.Context((4, 4, 4, 4))
    c.mt_load_params(mt_params)
    c.mt_seed(4321)
    c.mt_init(4096 * per_g, 4096 * per_u)
    m = oracle.mt_new(mt_params, seeds=gfx.glibc_rand(4321, 4096).astype(np.uint32))
    og, ou = oracle.mt_init_fields(m, per_g, per_u)
    for step in range(3):
        g, u, st, sd = c.mt_read()
        assert np.array_equal(u, ou), step
        assert np.array_equal(st.T.reshape(-1), np.ctypeslib.as_array(m.status)), step
        assert np.array_equal(sd, np.ctypeslib.as_array(m.seed)), step
        assert np.max(np.abs(g - og)) < 2e-4, step  # as the parity test of the bank
        c.mt_update()
        og, ou = oracle.mt_update_fields(m, per_g, per_u)
    c.close()
