"""The tuner where the FP64 sweeps run in fixed point: it chooses only among launches that differ,
leaves the FP64 link layout alone, and takes no settings from before."""
import numpy as np
import pytest

from conftest import haar, smooth_links

pytestmark = pytest.mark.gpu


def _context(gfx, dims, link_reals=12, scale=1.0):
    c = gfx.Context(dims, link_reals=link_reals)
    c.set_links(scale * smooth_links(dims, 0.4, 81))
    c.set_trafo(haar(int(np.prod(dims)), 82))
    return c


@pytest.mark.parametrize("link_reals", [12, 18])
def test_choices(gfx, link_reals):
    # one thread a site: blocks of 64 and 128, the odd half-sweep forwards or backwards
    for _ in range(4):
        c = _context(gfx, (12, 12, 12, 12), link_reals)
        t = c.autotune()
        assert t["link_reals64"] == link_reals
        assert t["block"][1] in (64, 128) and t["staging"][1] in (0, 2)
        assert t["sweep_ms"][1] > 0
        c.close()
    # four threads a site: nothing to choose
    c = _context(gfx, (4, 4, 6, 8), link_reals)
    c.set_tuning(block=(96, 96), staging=(1, 1))
    t = c.autotune()
    assert (t["block"][1], t["staging"][1], t["link_reals64"]) == (96, 1, link_reals)
    c.close()
    # links that keep to the FP64 kernels
    c = _context(gfx, (4, 4, 6, 8), link_reals, scale=1.5)
    t = c.autotune()
    assert t["block"][1] in (64, 128, 192, 256) and t["link_reals64"] in (12, 18)
    c.close()


def test_settings_of_the_fp64_kernels_are_not_taken(gfx, tmp_path):
    path = tmp_path / "tune.txt"
    c = _context(gfx, (4, 4, 6, 8))
    c.autotune(cache_path=str(path))
    c.close()
    key, rest = path.read_text().rstrip("\n").split("\t")
    assert key.endswith("|fx")
    fields = rest.split()
    fields[7] = "123.0"  # sweep_ms of FP64
    path.write_text(key[:-3] + "\t" + " ".join(fields) + "\n")
    c = _context(gfx, (4, 4, 6, 8))
    assert c.autotune(cache_path=str(path))["sweep_ms"][1] < 123.0
    c.close()
    # and its own are
    lines = path.read_text().splitlines()
    assert len(lines) == 2 and lines[1].startswith(key + "\t")
    path.write_text(key + "\t" + " ".join(fields) + "\n")
    c = _context(gfx, (4, 4, 6, 8))
    assert c.autotune(cache_path=str(path))["sweep_ms"][1] == 123.0
    c.close()
