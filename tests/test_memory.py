"""Buffers that a context takes only where there is room (the fixed-point fields of the FP64
sweeps, the random fields in reserve) are given back when a later call needs their memory."""
import numpy as np
import pytest

from conftest import haar, smooth_links

pytestmark = pytest.mark.gpu

DIMS = (24, 24, 24, 24)
V = 24 ** 4
MB = 1 << 20
FIXED = 720 * V    # fixed-point links and g
RESERVE = 160 * V  # two more pairs of the random fields below
# memory that a call is left with, and what it takes for good: get_links has a scratch of 576
# bytes a site, a change of layout a second link field beside it
CALLS = {"get_links": (200 * V, 576 * V), "layout": (700 * V, 768 * V),
         "random fields": (200 * V, 576 * V)}


def _fill(torch, leave):
    """device memory but for `leave` bytes, in pieces; kept while the list is"""
    torch.cuda.empty_cache()
    held = []
    while True:
        free = torch.cuda.mem_get_info()[0] - leave
        if free < 4 * MB:
            return held
        try:
            held.append(torch.empty(min(free, 64 << 30) // MB * MB, dtype=torch.uint8,
                                    device="cuda"))
        except torch.cuda.OutOfMemoryError:
            return held


@pytest.mark.parametrize("call", CALLS)
def test_optional_buffers_make_way(gfx, mt_params, call):
    torch = pytest.importorskip("torch")
    u, g = gfx.pinned_empty((4 * V, 3, 3, 2)), gfx.pinned_empty((V, 3, 3, 2))
    u.reshape(-1, 18)[:] = smooth_links(DIMS, 0.4, 71)
    g.reshape(-1, 18)[:] = haar(V, 72)
    out = gfx.pinned_empty((V, 3, 3, 2))
    held = []

    def run(full):
        c = gfx.Context(DIMS, link_reals=12)
        c.set_links(u)  # page-locked: no scratch
        c.set_trafo(g)
        if call == "random fields":
            c.mt_load_params(mt_params)
            c.mt_seed(73)
            c.mt_init(4 * V, 16 * V)  # 80 bytes a site, and as much twice in reserve
        held.extend(_fill(torch, FIXED + RESERVE + CALLS[call][0] + 32 * MB) if full else [])
        if call == "random fields":
            c.simanneal(0.5, 0.5, 2, expo=0.0)
        c.or_sweeps(3, 1.7, precision=1)
        bytes_taken = gfx.lib.gfx_device_bytes(c.handle)
        if full:
            held.extend(_fill(torch, CALLS[call][0]))
        if call == "layout":
            c.set_tuning(block=(128, 128), staging=(2, 2), link_reals64=18)
        links = c.get_links()
        if full:
            gone = FIXED + (RESERVE if call == "random fields" else 0)
            assert gfx.lib.gfx_device_bytes(c.handle) <= bytes_taken + CALLS[call][1] - gone + MB
        c.or_sweeps(1, 1.7, precision=1)
        c.get_trafo_into(out)
        c.close()
        return links, out.copy()

    try:
        (la, ga), (lb, gb) = run(False), run(True)
    finally:
        held.clear()  # a failure's traceback would keep it
        torch.cuda.empty_cache()
    assert np.array_equal(la, lb)
    # the last sweep of the second may be on the FP64 kernels: within 1e-13 of them
    assert np.max(np.abs(ga - gb)) < 1e-12


def test_batch_fields_make_way(gfx):
    # a batch polished in FP64, then with the rebased polish, whose fields need the memory
    torch = pytest.importorskip("torch")
    dims, n, v = (16, 16, 16, 16), 4, 16 ** 4
    b = gfx.Batch([dims], [n])
    b.set_links(0, smooth_links(dims, 0.25, 74))
    fixed = 576 * v + n * 144 * v       # links, and g of every copy
    rebased = n * (96 * 2 + 112) * v + 96 * 2 * v
    kw = dict(maxit=5000, eps=1e-12, checkinterval=20, omega=1.7, criterion=gfx.CRIT_THETA,
              checkinterval_double=2)
    held = []
    try:
        held.extend(_fill(torch, fixed + rebased // 2 + 32 * MB))
        free = torch.cuda.mem_get_info()[0]
        b.random_haar(75)
        first, _ = b.overrelax(gfx.Context.or_params(polish=0, **kw))
        assert free - torch.cuda.mem_get_info()[0] > fixed // 2  # taken
        held.extend(_fill(torch, rebased // 2 + 16 * MB))
        b.random_haar(75)
        second, _ = b.overrelax(gfx.Context.or_params(polish=2, **kw))
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert all(r["converged"] for r in first + second)
    for x, y in zip(first, second):
        assert abs(x["F"] - y["F"]) < 1e-9
    b.close()
