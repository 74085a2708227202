"""The FP64-accurate sweeps in 64-bit fixed point (gfx_fixed.cuh, gfx_fixed.cu): the
arithmetic on the CPU against long double and FP64, the kernels against the oracle where
they can go wrong, and the inputs that have to keep to the FP64 kernels."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

from conftest import haar, smooth_links

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("check,cases", [("fixed_check", 5000), ("fixed_kp_check", 50000)])
def test_fixed_point_errs_no_more_than_fp64(tmp_path, check, cases):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / check
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I", str(ROOT / "cudagfx_gb300" / "csrc"),
                    str(ROOT / "tests" / (check + ".cpp")), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(cases)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def _g12(g):
    return np.ascontiguousarray(np.asarray(g).reshape(-1, 18)[:, :12])


def _context(gfx, dims, u, g, link_reals=12, precision=0):
    c = gfx.Context(dims, precision=precision, link_reals=link_reals)
    c.set_links(u)
    c.set_trafo(g)
    return c


# 2^4: 8 sites a parity, less than a warp; 2x2x2x6: extents that wrap onto themselves;
# 4x6x10x6: a last block of 80 sites; 16x16x8x10: 80 whole blocks of 128
@pytest.mark.gpu
@pytest.mark.parametrize("link_reals,gauge", [(12, 0), (18, 1)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 2, 2, 6), (4, 6, 10, 6), (16, 16, 8, 10)])
def test_sweep_and_functional_at_tile_edges(gfx, oracle, dims, link_reals, gauge):
    V = int(np.prod(dims))
    u, g = smooth_links(dims, 0.6, 11), haar(V, 12)
    c = _context(gfx, dims, u, g, link_reals)
    lat, gf12, g12 = oracle.lattice(dims), oracle.to2v(u), _g12(g)
    ndir = 3 if gauge else 4
    for _ in range(2):
        for parity in (0, 1):
            c.or_halfsweep(parity, omega=1.7, gauge=gauge, precision=1)
            oracle.or_halfsweep(lat, gf12, g12, parity, 1.7, ndir)
    # one FP64 half-sweep is within 1e-13 of the oracle on such fields; four of them
    f = c.functional(gauge=gauge, precision=1)
    assert np.max(np.abs(_g12(c.get_trafo()) - g12)) < 4e-13
    o = oracle.functional(lat, gf12, g12, ndir)
    assert f.F == pytest.approx(o["F"], rel=1e-12)
    assert f.dAdA == pytest.approx(o["dAdA"], rel=1e-11)
    assert f.maxdAdA == pytest.approx(o["maxdAdA"], rel=1e-11)
    c.close()


# the functional straight from FP64 fields (converted site by site): the same lattices, and
# links and g outside the bounds, whose sites are measured in FP64
@pytest.mark.gpu
@pytest.mark.parametrize("scale_u,scale_g", [(1.0, 1.0), (1.5, 1.0), (1.0, 0.75)])
@pytest.mark.parametrize("link_reals,gauge", [(12, 0), (18, 1)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 6, 10, 6), (16, 16, 8, 10)])
def test_functional_of_fp64_fields(gfx, oracle, dims, link_reals, gauge, scale_u, scale_g):
    V = int(np.prod(dims))
    u, g = smooth_links(dims, 0.6, 13), haar(V, 14)
    # some matrices only, rows 0, 1 (row 2 as the 12-real layout rebuilds it)
    u[::7, :12] *= scale_u
    u[::7, 12:] *= scale_u * scale_u
    g[::5, :12] *= scale_g
    c = _context(gfx, dims, u, g, link_reals)
    f = c.functional(gauge=gauge, precision=1)
    o = oracle.functional(oracle.lattice(dims), oracle.to2v(u), _g12(g), 3 if gauge else 4)
    assert f.F == pytest.approx(o["F"], rel=1e-12)
    assert f.dAdA == pytest.approx(o["dAdA"], rel=1e-12)
    assert f.maxdAdA == pytest.approx(o["maxdAdA"], rel=1e-12)
    c.close()


# partial last blocks, extents that wrap onto themselves, and links measured in FP64
@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 1.5])
@pytest.mark.parametrize("link_reals", [12, 18])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 6, 10, 6), (16, 16, 8, 10)])
def test_plaquette(gfx, oracle, dims, link_reals, scale):
    u = smooth_links(dims, 0.6, 15)
    u[::7, :12] *= scale
    u[::7, 12:] *= scale * scale
    c = gfx.Context(dims, link_reals=link_reals)
    c.set_links(u)
    # a sum of 18 terms below 1 per plane and site in fixed point or FP64: 1e-14 of a value
    # that is at least 1e-2 here
    want = oracle.plaquette(oracle.lattice(dims), oracle.to2v(u))
    assert c.plaquette() == pytest.approx(want, rel=1e-13)
    c.close()


@pytest.mark.gpu
def test_reading_g_does_not_change_the_run(gfx):
    # get_trafo and functional between sweeps leave the bits of the run as they are
    dims = (8, 8, 8, 12)
    u, g = smooth_links(dims, 0.4, 3), haar(int(np.prod(dims)), 4)
    a, b = _context(gfx, dims, u, g), _context(gfx, dims, u, g)
    a.or_sweeps(6, 1.7, precision=1)
    for _ in range(3):
        b.or_sweeps(2, 1.7, precision=1)
        b.functional()
        b.get_trafo()
    assert np.array_equal(a.get_trafo(), b.get_trafo())
    # and a g that is set again is the one that is used
    b.set_trafo(g)
    b.or_sweeps(6, 1.7, precision=1)
    assert np.array_equal(a.get_trafo(), b.get_trafo())
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["scaled links", "omega", "start"])
def test_inputs_outside_the_bounds_take_the_fp64_kernels(gfx, oracle, case):
    dims = (4, 4, 6, 8)
    V = int(np.prod(dims))
    u, g, omega = smooth_links(dims, 0.4, 21), haar(V, 22), 1.7
    lat = oracle.lattice(dims)
    if case == "scaled links":  # entries up to 2.5, far from unitary
        u = 2.5 * u
    elif case == "omega":
        omega = 2.25
    else:  # a start read from 32-bit data: unitary to 1e-7, so the first sweep is FP64
        g = g.astype(np.float32).astype(np.float64)
    a = _context(gfx, dims, u, g)
    a.or_sweeps(3, omega, precision=1)
    got = _g12(a.get_trafo())
    if case == "start":
        b = _context(gfx, dims, u, g)
        for _ in range(3):
            b.or_sweeps(1, omega, precision=1)
        assert np.max(np.abs(got - _g12(b.get_trafo()))) < 3e-13
        b.close()
    else:
        gf12, g12 = oracle.to2v(u), _g12(g)
        for _ in range(3):
            for parity in (0, 1):
                oracle.or_halfsweep(lat, gf12, g12, parity, omega)
        assert np.max(np.abs(got - g12)) < 1e-12
    a.close()


# a Kennedy-Pendleton chain in fixed point against the FP64 kernel's half-sweeps with the same
# random numbers: lattices as above; beta below the arithmetic's bound and links far from
# unitary, which keep to the FP64 kernel.  A link errs by some 1e-15 of FP64 rounding per
# update, amplified a few times by each of the later updates of a sweep.
@pytest.mark.gpu
@pytest.mark.parametrize("dims,link_reals,beta,scale",
                         [((2, 2, 2, 2), 12, 6.0, 1.0), ((2, 2, 2, 6), 18, 6.0, 1.0),
                          ((4, 6, 10, 6), 12, 5.7, 1.0), ((16, 16, 8, 10), 18, 6.2, 1.0),
                          ((4, 4, 6, 8), 12, 3.0, 1.0), ((4, 4, 6, 8), 12, 6.0, 1.5)])
def test_link_heatbath_chain(gfx, mt_params, dims, link_reals, beta, scale):
    V = int(np.prod(dims))
    u = smooth_links(dims, 0.6, 17)
    u[::7, :12] *= scale
    u[::7, 12:] *= scale * scale
    per = 4096 * 38

    def make():
        c = gfx.Context(dims, link_reals=link_reals)
        c.set_links(u)
        c.mt_load_params(mt_params)
        c.mt_seed(91)
        c.mt_init(-(-2 * V // per) * per, -(-8 * V // per) * per)
        return c

    a, b = make(), make()
    a.thermalize(beta, 1, variant=gfx.HB_KENNEDY_PENDLETON)
    for nu in range(4):
        for parity in (0, 1):
            b.link_heatbath_halfsweep(parity, nu, beta, variant=gfx.HB_KENNEDY_PENDLETON)
            b.mt_update()
    x, y = a.get_links(), b.get_links()
    if beta < 3.75 or scale != 1.0:
        assert np.array_equal(x, y)
    else:
        assert np.max(np.abs(x - y)) < 1e-11
        # a chain in several calls is the chain of one
        a.thermalize(beta, 3, variant=gfx.HB_KENNEDY_PENDLETON)
        c = make()
        for n in (1, 1, 2):
            c.thermalize(beta, n, variant=gfx.HB_KENNEDY_PENDLETON)
        assert np.array_equal(a.get_links(), c.get_links())
        c.close()
    a.close()
    b.close()
