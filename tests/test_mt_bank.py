"""The twister bank's kernel at the edges of its steps (ten outputs of a twister), tiles (160)
and ring (19): bit-exact uniforms, states and seeds against the oracle over several updates;
and runs of heatbath steps with the updates made ahead of them."""
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


# a run of steps makes the next fields while the current ones are in use: the same chain, the
# same bank and the same fields as one call per step
def test_runs_leave_the_fields_of_single_steps(gfx, mt_params):
    dims = (4, 4, 6, 8)
    V = int(np.prod(dims))

    def make():
        c = gfx.Context(dims, precision=gfx.PREC_MIXED)
        c.set_links(gfx.random_init_haar(5, 4 * V))
        c.set_trafo(gfx.random_init_haar(6, V))
        c.mt_load_params(mt_params)
        c.mt_seed(77)
        c.mt_init(4096 * 6, 4096 * 10)
        return c

    a, b = make(), make()
    p = gfx.SAParams(0.3, 0.3, 0.0, 7, 100, 1)  # one temperature, seven steps
    a._check(gfx.lib.gfx_simanneal_range(a.handle, p, 0, 7))
    for k in range(7):
        b._check(gfx.lib.gfx_simanneal_range(b.handle, p, k, 1))
    a.thermalize(6.0, 3, variant=gfx.HB_KENNEDY_PENDLETON)
    for _ in range(3):
        b.thermalize(6.0, 1, variant=gfx.HB_KENNEDY_PENDLETON)
    assert np.array_equal(a.get_trafo(), b.get_trafo())
    assert np.array_equal(a.get_links(), b.get_links())
    for x, y in zip(a.mt_read(), b.mt_read()):
        assert np.array_equal(x, y)
    # fields of other sizes after a run
    a.mt_init(4096 * 8, 4096 * 20)
    b.mt_init(4096 * 8, 4096 * 20)
    a.simanneal(0.3, 0.3, 2, expo=0.0)
    b.simanneal(0.3, 0.3, 2, expo=0.0)
    for x, y in zip(a.mt_read(), b.mt_read()):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("steps", [1, 2, 5])
@pytest.mark.parametrize("precision", ["PREC_DOUBLE", "PREC_MIXED"])
def test_run_is_half_sweeps_and_updates(gfx, mt_params, precision, steps):
    # a run's updates are made ahead of its steps, fewer of them than fields in reserve or more
    dims = (4, 6, 4, 10)
    V = int(np.prod(dims))
    T = 0.25

    def make():
        c = gfx.Context(dims, precision=getattr(gfx, precision))
        c.set_links(gfx.random_init_haar(8, 4 * V))
        c.set_trafo(gfx.random_init_haar(9, V))
        c.mt_load_params(mt_params)
        c.mt_seed(31)
        c.mt_init(4096 * 2, 4096 * 6)
        return c

    a, b = make(), make()
    a._check(gfx.lib.gfx_simanneal_range(a.handle, gfx.SAParams(T, T, 0.0, steps, 100, 0), 0,
                                         steps))
    for _ in range(steps):
        for parity in (0, 1):
            b.sa_halfsweep(parity, 1.0 / T, 1 if precision == "PREC_DOUBLE" else 0)
            b.mt_update()
    assert np.array_equal(a.get_trafo(), b.get_trafo())
    for x, y in zip(a.mt_read(), b.mt_read()):
        assert np.array_equal(x, y)
    a.close()
    b.close()
