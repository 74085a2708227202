"""The memory of large results (cudagfx_gb300._Results): kept for the next one of its size only
after the last view of a result is gone, bounded, and given back on close."""
import gc
import threading

import numpy as np
import pytest

from cudagfx_gb300 import _Results

LEAST = _Results.LEAST // 8


def _at(a):
    return a.__array_interface__["data"][0]


@pytest.mark.parametrize("n,kept", [(LEAST - 1, False), (LEAST, True), (LEAST + 1, True)])
def test_reuse(n, kept):
    r = _Results()
    a = r.empty((n,))
    assert a.shape == (n,) and a.dtype == np.float64 and a.flags.writeable and a.flags.c_contiguous
    at = _at(a)
    view = a[3:5].reshape(2, 1)
    a[:] = 1.0
    del a
    gc.collect()
    b = r.empty((n,))  # the view holds the first block
    b[:] = 2.0
    assert view[0, 0] == 1.0 and not np.shares_memory(b, view)
    del view
    gc.collect()
    if kept:
        c = r.empty((n,))
        assert _at(c) == at
        assert not np.shares_memory(c, b)


def test_bounded_and_given_back():
    r = _Results()
    a = [r.empty((LEAST, 2)) for _ in range(4)]
    assert len({_at(x) for x in a}) == 4
    other = r.empty((LEAST + 7,))
    del a, other
    gc.collect()
    assert sorted(len(k) for k in r._kept.values()) == [1, 1]
    late = r.empty((LEAST, 2))
    late[:] = 5.0
    r.close()
    assert all(len(k) == 0 for k in r._kept.values())
    assert late.sum() == 10.0 * LEAST  # a result outlives its context
    del late
    gc.collect()
    assert all(len(k) == 0 for k in r._kept.values())
    assert r.empty((LEAST,)).base is None


def test_largest():
    r = _Results()
    assert r.empty((_Results.MOST // 8 + 1,)).base is None  # never written, so never backed
    assert not r._kept


def test_threads():
    r = _Results()
    bad = []

    def work(k):
        for i in range(10):
            a = r.empty((LEAST,))
            a[:] = 100 * k + i
            b = a[::1024]
            del a
            if not (b == 100 * k + i).all():
                bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
