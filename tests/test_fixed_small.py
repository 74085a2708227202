"""The fixed-point update where norms are small (a star, a projection or a row that nearly
vanishes): the arithmetic on the CPU, and both kernels of the half-sweep on such fields."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

from conftest import haar, smooth_links, su3_from_rows

ROOT = pathlib.Path(__file__).resolve().parent.parent


def test_small_norms_keep_fp64_accuracy(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "fixed_small_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I", str(ROOT / "cudagfx_gb300" / "csrc"),
                    str(ROOT / "tests" / "fixed_small_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "1000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def _cplx(m):
    m = np.asarray(m).reshape(-1, 3, 3, 2)
    return m[..., 0] + 1j * m[..., 1]


def _real(m):
    return np.stack([m.real, m.imag], -1).reshape(-1, 18)


def _transformed(dims, phases, noise, seed):
    """links h(x)^+ P_mu N h(x+mu), of P_mu = diag(phases[mu]) and N near 1, and g = h"""
    lx, ly, lz, lt = dims
    V = lx * ly * lz * lt
    h = _cplx(haar(V, seed)).reshape(lt, lz, ly, lx, 3, 3)
    rng = np.random.default_rng(seed + 1)
    u = np.empty((lt, lz, ly, lx, 4, 3, 3), complex)
    for mu in range(4):
        rows = np.zeros((V, 2, 3), complex)
        rows[:, 0, 0] = rows[:, 1, 1] = 1.0
        rows += noise * (rng.normal(size=rows.shape) + 1j * rng.normal(size=rows.shape))
        n = _cplx(su3_from_rows(rows)).reshape(h.shape)
        p = np.diag(np.asarray(phases[mu], complex))
        u[..., mu, :, :] = np.conj(np.swapaxes(h, -1, -2)) @ p @ n @ np.roll(h, -1, 3 - mu)
    return _real(u.reshape(-1, 3, 3)), _real(h.reshape(-1, 3, 3))


FLIP = [(-1, -1, 1)] * 4                                          # S = diag(-1, -1, 1)
CENTRE = [(np.exp(2j * np.pi * k / 3),) * 3 for k in range(3)] + [(1, 1, 1)]  # sums to 0


def _off_unitary(g):
    m = _cplx(g)[:, :2]
    return np.max(np.abs(np.einsum("nik,njk->nij", m, np.conj(m)) - np.eye(2)))


# four threads a site, and one thread a site (more than 9,728 sites of a parity).  With
# r = 1 - 4 omega + 2 omega^2 = -3.0e-4 at omega 1.707 the distance of the start from unitary and
# the rows' rounding, 4e-16, count 1/r times in either
@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(4, 4, 6, 8), (12, 12, 12, 12)])
def test_overrelaxed_rows_that_nearly_vanish(gfx, oracle, dims):
    u, g = _transformed(dims, FLIP, 0.0, 51)
    c = gfx.Context(dims)
    c.set_links(u)
    c.set_trafo(g)
    g12 = np.ascontiguousarray(g[:, :12])
    lat, gf12 = oracle.lattice(dims), oracle.to2v(u)
    bound = 2 * (_off_unitary(g) + 4e-16) / 3.0e-4
    c.or_halfsweep(0, omega=1.707, precision=1)
    oracle.or_halfsweep(lat, gf12, g12, 0, 1.707)
    got = c.get_trafo().reshape(-1, 18)
    assert np.max(np.abs(got[:, :12] - g12)) < bound
    t, z, y, x = np.indices(dims[::-1])
    assert _off_unitary(got[((t + z + y + x) % 2 == 0).reshape(-1)]) < 2e-15
    c.close()


# the same fields on 8^4 (four threads a site) and repeated over 16^4 (one thread): the same bits
@pytest.mark.gpu
@pytest.mark.parametrize("gauge", [0, 1])
@pytest.mark.parametrize("fields", ["smooth", "flip", "centre"])
def test_both_kernels_give_the_same_bits(gfx, gauge, fields):
    dims, twice = (8, 8, 8, 8), (16, 16, 16, 16)
    V = 8 ** 4
    if fields == "smooth":
        u, g = smooth_links(dims, 0.5, 61), haar(V, 62)
    else:
        u, g = _transformed(dims, FLIP if fields == "flip" else CENTRE, 1e-5, 63)

    def tiled(f):
        f = f.reshape(8, 8, 8, 8, -1)
        return np.ascontiguousarray(np.tile(f, (2, 2, 2, 2, 1)))

    out = []
    for d, uu, gg in ((dims, u, g), (twice, tiled(u), tiled(g))):
        c = gfx.Context(d, link_reals=18)
        c.set_links(uu)
        c.set_trafo(gg)
        c.or_sweeps(3, 1.707, gauge=gauge, precision=1)
        out.append(c.get_trafo())
        c.close()
    assert np.array_equal(tiled(out[0]).reshape(-1), out[1].reshape(-1))
