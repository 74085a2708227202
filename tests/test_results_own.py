"""Large results are ordinary arrays: they own their data, can be resized in place, and leave the
thread's numpy memory handler as it was."""
import gc

import numpy as np
import pytest

from cudagfx_gb300 import _Results

N = _Results.LEAST // 8


def _at(a):
    return a.__array_interface__["data"][0]


@pytest.mark.parametrize("shape", [(N,), (N // 18, 3, 3, 2)])
def test_results_own_their_data(shape):
    n = int(np.prod(shape)) + 18  # of the second shape: a size of its own above the least
    shape = shape if len(shape) == 1 else (n // 18 + 1, 3, 3, 2)
    r = _Results()
    for _ in range(2):  # fresh and kept memory
        a = r.empty(shape)
        assert a.flags.owndata and a.base is None and type(a) is np.ndarray and a.shape == shape
        del a
        gc.collect()
    a = r.empty(shape)
    a[:] = 3.0
    a.resize((a.size // 2,), refcheck=False)
    assert a.shape[0] * 2 <= int(np.prod(shape)) and (a == 3.0).all()
    a.resize((N + 4096,), refcheck=False)
    assert a.size == N + 4096 and a[0] == 3.0
    del a
    gc.collect()
    assert [k for k in r._kept if k == N + 4096]
    r.close()
    assert not r._kept


def test_other_arrays_are_numpys():
    r = _Results()
    a = r.empty((N,))
    b, c = np.empty(N), a.copy()
    del b, c
    gc.collect()
    assert not r._kept
    at = _at(a)
    del a
    gc.collect()
    assert r._kept == {N: [at]}
    d = np.empty(N)  # not from the pool
    assert r._kept == {N: [at]} and _at(d) != at
    with pytest.raises(TypeError):
        r.empty(("a",))
    r.close()


def test_pool_outlives_its_owner():
    r = _Results()
    a, b = r.empty((N,)), r.empty((N,))
    a[:] = 1.0
    b[:] = 2.0
    del r
    gc.collect()
    assert a.sum() == N and b.sum() == 2 * N
    del a, b
    gc.collect()
