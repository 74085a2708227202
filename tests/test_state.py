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


def _chain(gfx, dims, mt_params, link_reals):
    V = int(np.prod(dims))
    c = _context(gfx, dims, smooth_links(dims, 0.5, 33), haar(V, 34), link_reals=link_reals)
    c.mt_load_params(mt_params)
    c.mt_seed(35)
    per = 4096 * 38  # whole rounds: a stream that goes on from call to call
    c.mt_init(-(-2 * V // per) * per, -(-8 * V // per) * per)
    return c


# four threads a site, and one thread a site (more than 9,728 sites of a parity)
DIMS = [(4, 4, 6, 8), (12, 12, 12, 12)]


@pytest.mark.parametrize("link_reals", [12, 18])
@pytest.mark.parametrize("dims", DIMS)
def test_reading_saving_and_setting_do_not_change_the_run(gfx, mt_params, tmp_path, dims,
                                                          link_reals):
    plain, read, saved, again = (_chain(gfx, dims, mt_params, link_reals) for _ in range(4))
    path = str(tmp_path / "state")
    cs = (plain, read, saved, again)

    def between():
        read.get_links(), read.get_trafo(), read.plaquette(), read.functional()
        saved.checkpoint_save(path)
        again.set_links(again.get_links())
        again.set_trafo(again.get_trafo())

    for _ in range(2):
        for c in cs:
            c.thermalize(6.0, 1, variant=gfx.HB_KENNEDY_PENDLETON)
        between()
        for c in cs:
            c.or_sweeps(2, 1.7, precision=1)
        between()
    for c in cs:
        c.or_sweeps(2, 1.7, gauge=gfx.COULOMB, precision=1)
    restored = _chain(gfx, dims, mt_params, link_reals)
    restored.checkpoint_load(path)
    restored.or_sweeps(2, 1.7, gauge=gfx.COULOMB, precision=1)
    for c in cs[1:] + (restored,):
        assert np.array_equal(c.get_links(), plain.get_links())
        assert np.array_equal(c.get_trafo(), plain.get_trafo())
        c.close()
    plain.close()


@pytest.mark.parametrize("link_reals", [12, 18])
@pytest.mark.parametrize("gauge", [0, 1])
@pytest.mark.parametrize("dims", DIMS)
def test_functional_of_the_same_fields_has_the_same_bits(gfx, dims, gauge, link_reals):
    # as the sweeps left the fields, after reading g, set again, and in a new context
    u, g = smooth_links(dims, 0.5, 36), haar(int(np.prod(dims)), 37)
    a = _context(gfx, dims, u, g, link_reals=link_reals)
    a.or_sweeps(3, 1.7, gauge=gauge, precision=1)
    f = [a.functional(gauge).as_dict()]
    last = a.get_trafo()
    f.append(a.functional(gauge).as_dict())
    a.set_trafo(last)
    f.append(a.functional(gauge).as_dict())
    b = _context(gfx, dims, u, last, link_reals=link_reals)
    f.append(b.functional(gauge).as_dict())
    r = a.overrelax(maxit=30, eps=1e-30, checkinterval=7, omega=1.7, criterion=gfx.CRIT_THETA,
                    gauge=gauge)
    b.set_trafo(a.get_trafo())
    assert all(x == f[0] for x in f[1:])
    # the solve's last check is 1 + 4 * 7 sweeps in, its tail one sweep further
    b.set_trafo(last)
    b.or_sweeps(1 + 4 * 7, 1.7, gauge=gauge, precision=1)
    assert b.functional(gauge).F == r.final_values.F
    assert b.functional(gauge).theta == r.final_values.theta
    a.close()
    b.close()


@pytest.mark.parametrize("dims", DIMS)
def test_sites_that_are_not_updated_keep_their_bits(gfx, dims):
    # g near the identity: small entries have digits far below those of the fixed-point fields
    V = int(np.prod(dims))
    u, g = smooth_links(dims, 0.5, 38), smooth_links(dims, 1e-6, 39)[:V]
    c = _context(gfx, dims, u, g)
    before = c.get_trafo().reshape(V, 18)
    c.or_sweeps(0, 1.7, precision=1)
    assert np.array_equal(c.get_trafo().reshape(V, 18), before)
    t, z, y, x = np.indices(dims[::-1])
    even = ((t + z + y + x) % 2 == 0).reshape(-1)
    c.or_halfsweep(1, omega=1.7, precision=1)
    after = c.get_trafo().reshape(V, 18)
    assert np.array_equal(after[even], before[even])
    assert not np.any(np.all(after[~even] == before[~even], axis=1))
    c.or_halfsweep(0, omega=1.7, precision=1)
    both = c.get_trafo().reshape(V, 18)
    assert np.array_equal(both[~even], after[~even])
    c.close()


@pytest.mark.parametrize("polish", [0, 1, 2])
def test_a_solve_again(gfx, polish):
    # the loop graphs of the first solve serve the second
    dims = (4, 4, 6, 8)
    u, g = smooth_links(dims, 0.4, 40), haar(int(np.prod(dims)), 41)
    c = _context(gfx, dims, u, g, precision=gfx.PREC_MIXED)
    out = []
    for _ in range(2):
        c.set_trafo(g)
        r = c.overrelax(maxit=5000, eps=1e-14, checkinterval=10, omega=1.7,
                        criterion=gfx.CRIT_THETA, polish=polish)
        assert r.converged and r.sweeps_double > 0
        f = c.functional()
        assert f.theta < 1e-14
        out.append((r.iterations, f.F, c.get_trafo()))
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])
    c.close()


@pytest.mark.parametrize("link_reals", [12, 18])
@pytest.mark.parametrize("variant,beta", [(1, 6.0), (1, 3.0), (0, 6.0)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 6), (4, 6, 10, 6)])
def test_a_chain_is_its_half_sweeps(gfx, mt_params, dims, variant, beta, link_reals):
    a, b = (_chain(gfx, dims, mt_params, link_reals) for _ in range(2))
    for _ in range(2):
        a.thermalize(beta, 1, variant=variant)
        for nu in range(4):
            for parity in (0, 1):
                b.link_heatbath_halfsweep(parity, nu, beta, variant=variant)
                b.mt_update()
        assert np.array_equal(a.get_links(), b.get_links())
        assert a.plaquette() == b.plaquette()
    a.close()
    b.close()
