"""Result arrays from recycled host memory when meshes come and go (no GPU): closing one leaves the
other meshes' blocks, the next mesh's first results find them, and what is kept is bounded."""
import gc
import random
import threading
import tracemalloc

import numpy as np
import pytest

from ufemism_gb300 import api


class _Library:
    """Stands in for the native library where a handle is only closed."""

    def ufe_mesh_destroy(self, h):
        return 0

    def ufe_batch_destroy(self, h):
        return 0


def handle(kind):
    h = kind.__new__(kind)
    h._h = 1
    api._pool.opened()
    return h


@pytest.fixture
def pool(monkeypatch):
    p = api._HostPool(limit=64 << 20, rest=16 << 20)
    monkeypatch.setattr(api, "_pool", p)
    monkeypatch.setattr(api.nat, "load", lambda: _Library())
    return p


@pytest.mark.parametrize("kind", [api.DeviceMesh, api.Batch])
@pytest.mark.parametrize("by_collection", [False, True])
def test_closing_a_handle_leaves_the_others_blocks(pool, kind, by_collection):
    kept, other = handle(api.DeviceMesh), handle(kind)
    used, idle = pool.array(200000), pool.array(300000)
    where = {used.ctypes.data, idle.ctypes.data}
    del idle
    gc.collect()
    if by_collection:
        del other
        gc.collect()
    else:
        other.close()
    del used   # in use when the other handle was closed
    gc.collect()
    assert {a.ctypes.data for a in [pool.array(200000), pool.array(300000)]} == where
    kept.close()


@pytest.mark.parametrize("factor", [0.8, 1.0])
def test_the_next_mesh_finds_the_blocks_of_the_last(pool, factor):
    mesh = handle(api.DeviceMesh)
    a = pool.group([(100000, 4), 100000, 50000])
    where = min(x.ctypes.data for x in a)
    del a
    mesh.close()   # the only one
    gc.collect()
    handle(api.DeviceMesh)
    n = int(100000 * factor)
    assert min(x.ctypes.data for x in pool.group([(n, 4), n, n // 2])) == where


def test_idle_memory_after_the_last_handle_is_bounded(pool):
    mesh, batch = handle(api.DeviceMesh), handle(api.Batch)
    arrays = [pool.array(1 << 20) for _ in range(12)]   # 8 MiB each
    last = arrays[-1].ctypes.data
    for _ in range(12):
        arrays.pop(0)
    gc.collect()
    assert 16 << 20 < pool._bytes <= 64 << 20
    mesh.close()
    assert 16 << 20 < pool._bytes
    batch.close()
    assert 0 < pool._bytes <= 16 << 20
    assert pool.array(1 << 20).ctypes.data == last   # the blocks used last are the ones kept


def test_a_block_beyond_the_limit_leaves_the_others(pool):
    mesh = handle(api.DeviceMesh)
    a = pool.array(1 << 20)
    where = a.ctypes.data
    del a
    b = pool.array(16 << 20)   # 128 MiB
    del b
    gc.collect()
    assert pool._bytes == 8 << 20 and pool.array(1 << 20).ctypes.data == where
    mesh.close()


def test_a_handle_collected_inside_the_pool_does_not_wait_for_itself(pool):
    mesh, array = handle(api.DeviceMesh), pool.array(100000)
    with pool._lock:   # a collection in the middle of the pool's work
        del mesh, array
        gc.collect()
    np.testing.assert_array_equal(pool.zeros(100000), 0.0)
    assert pool._open == 0


def test_a_lease_is_a_numpy_array_and_ends_once():
    """No Python-level buffer method, which the interpreter knows from 3.12 on only; the lease ends
    with the last view, also when that was made from a base of the array."""
    pool = api._HostPool()
    assert "__buffer__" not in vars(api._Lease)
    a = pool.array((5000, 20), order="F")
    assert type(a) is np.ndarray
    chain, x = [], a
    while isinstance(x, np.ndarray):
        chain.append(x)
        x = x.base
    views = [c[1:] for c in chain] + [c.view() for c in chain]
    del a, chain, x
    while views:
        assert pool._bytes == 0
        views.pop()
        gc.collect()
    assert pool._bytes == 13 << 16


@pytest.mark.parametrize("dtype", [np.float64, np.int32])
@pytest.mark.parametrize("keep", [0, 2, 5])
def test_a_kept_field_keeps_little_else(keep, dtype):
    """The fields of a result lie one after the other, yet a caller that keeps one field of each of
    many results keeps about these fields' memory (and the other fields are whole and apart)."""
    pool = api._HostPool()
    shapes = [(40000,), (20000, 2), (60000,), (7, 3000), (0,), (60001,)]
    tracemalloc.start()
    kept, biggest = [], 0
    for k in range(60):
        r = pool.group(shapes, dtype, "F")
        spans = sorted((a.ctypes.data, a.ctypes.data + a.nbytes) for a in r if a.size)
        assert all(x[1] <= y[0] for x, y in zip(spans, spans[1:]))
        assert [a.shape for a in r] == shapes and all(a.flags.f_contiguous for a in r)
        if k == 0:
            assert all(x[1] == y[0] for x, y in zip(spans, spans[1:]))
        for a in r:
            a[...] = k
        biggest = sum(a.nbytes for a in r)
        kept.append(r[keep])
        del r, a
    assert all(np.all(a == k) for k, a in enumerate(kept))
    assert tracemalloc.get_traced_memory()[0] < 1.5 * sum(a.nbytes for a in kept) + 3 * biggest
    tracemalloc.stop()
    del kept
    gc.collect()
    assert not pool._partial and pool._bytes == sum(b.size for b in pool._idle)


def test_ranges_join_again_in_any_order():
    rng = np.random.default_rng(5)
    block = api._Block(4096, 0)
    for _ in range(50):
        cuts = np.unique(np.concatenate([[0, 4096], rng.integers(1, 4096, 9)]))
        ranges = [(int(a), int(b)) for a, b in zip(cuts, cuts[1:])]
        for k in rng.permutation(len(ranges)):
            block.take(*ranges[k])
        assert block.free == []
        for k in rng.permutation(len(ranges)):
            block.give(*ranges[k])
        assert block.free == [(0, 4096)]


def test_stale_pages_are_written_in_the_range_only(monkeypatch):
    monkeypatch.setattr(api.time, "monotonic", iter(range(100)).__next__)   # a second between requests
    pool = api._HostPool()
    page = api.mmap.PAGESIZE
    a = pool.group([16 * page, 16 * page, 16 * page], np.uint8)
    for x in a:
        x.fill(7)
    middle = a.pop(1).ctypes.data
    b = pool.array(16 * page, np.uint8)
    assert b.ctypes.data == middle
    assert np.all(b[::page] == 0) and b[-1] == 0 and np.count_nonzero(b == 0) == 17
    assert all(np.all(x == 7) for x in a)


def test_of_many_blocks_one_of_the_size_is_found():
    pool = api._HostPool()
    sizes = [65536 * k for k in range(1, 40)]
    held = [pool.array(n, np.uint8) for n in sizes]
    where = [x.ctypes.data for x in held]
    del held
    for n, at in reversed(list(zip(sizes, where))):
        x = pool.array(n, np.uint8)
        assert x.ctypes.data == at
        del x
    pool.release()
    assert not pool._of_size and not pool._idle


def test_threads_hold_and_drop_fields_in_any_order():
    """Random groups (empty and small arrays among them), some fields kept, collections and releases in
    between: every field keeps its values while it is held, and the books balance in the end."""
    pool = api._HostPool(limit=24 << 20, rest=8 << 20)
    bad = []

    def work(k):
        rng, held = random.Random(k), []
        try:
            for i in range(300):
                shapes = [rng.choice([1000, 9000, 20000, 70001, (300, 100), (0,), 5]) for _ in range(rng.randint(1, 8))]
                fields = pool.group(shapes, rng.choice([np.float64, np.int32]), rng.choice("CF"))
                for a in fields:
                    a[...] = 1000 * k + i
                held.append((1000 * k + i, rng.sample(fields, rng.randint(0, len(fields)))))
                if len(held) > 12:
                    tag, kept = held.pop(rng.randrange(len(held)))
                    bad.extend(tag for a in kept if not np.all(a == tag))
                if rng.random() < 0.01:
                    pool.release()
                if rng.random() < 0.02:
                    gc.collect()
            bad.extend(tag for tag, kept in held if not all(np.all(a == tag) for a in kept))
        except Exception as e:
            bad.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    gc.collect()
    assert not bad
    assert not pool._partial and pool._bytes == sum(b.size for b in pool._idle) <= 8 << 20
    assert sum(map(len, pool._of_size.values())) == len(pool._idle)
    assert all(b.free == [(0, b.size)] for b in pool._idle)
