"""Result arrays from recycled host memory (no GPU): a block is handed out again only when no array
or view of it is left, idle memory is bounded and released, and threads never share a block."""
import gc
import threading

import numpy as np
import pytest

from ufemism_gb300 import api


@pytest.mark.parametrize("shape,dtype,order", [((8192,), np.float64, "C"), ((5000, 15), np.float64, "F"),
                                               ((40001,), np.int32, "C"), ((10,), np.float64, "C")])
def test_arrays_are_like_new_ones(shape, dtype, order):
    pool = api._HostPool()
    a = pool.zeros(shape, dtype, order)
    assert a.shape == shape and a.dtype == dtype and a.flags.writeable and not a.any()
    assert a.flags.f_contiguous if order == "F" else a.flags.c_contiguous
    a[...] = 3
    b = pool.array(shape, dtype, order)
    b[...] = 4
    assert np.all(a == 3)


def test_a_view_keeps_its_block():
    pool = api._HostPool()
    a = pool.zeros((4096, 4), order="F")
    view, where = a[100:200, 1], a.ctypes.data
    del a
    gc.collect()
    others = [pool.array((4096, 4), order="F") for _ in range(3)]
    for o in others:
        o[...] = 9
    assert not view.any() and where not in [o.ctypes.data for o in others]
    del view, o, others
    gc.collect()
    assert where in [x.ctypes.data for x in [pool.array((4096, 4), order="F") for _ in range(4)]]


def test_idle_memory_is_bounded_and_released():
    pool = api._HostPool(limit=1 << 20)
    arrays = [pool.array(65536) for _ in range(8)]   # 512 KiB each
    del arrays
    gc.collect()
    assert 0 < pool._bytes <= 1 << 20
    held = pool.array(65536)
    pool.release()
    assert pool._bytes == 0 and not pool._idle
    del held   # leased before the release: not kept
    gc.collect()
    assert pool._bytes == 0 and not pool._idle


def test_threads_do_not_share_blocks():
    pool = api._HostPool()
    bad = []

    def work(k):
        for i in range(300):
            a = pool.array(8192 + 8192 * (i % 3))
            a.fill(k)
            if not np.all(a == k):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
