"""The pool of page-locked result memory, with a library that hands out ordinary memory."""
import ctypes
import gc
import threading

import numpy
import pytest

pytest.importorskip("torch")
from orbkit_gb300 import hostmem  # noqa: E402


class Library:
    def __init__(self):
        self.live = {}

    def okg_host_alloc(self, size, p):
        buf = ctypes.create_string_buffer(size)
        p._obj.value = ctypes.addressof(buf)
        self.live[p._obj.value] = (buf, size)
        return 0

    def okg_host_free(self, p):
        del self.live[p.value]
        return 0

    def locked(self):
        return sum(s for _, s in self.live.values())


@pytest.fixture
def pool(monkeypatch):
    lib = Library()
    monkeypatch.setattr(hostmem._lib, "load", lambda: lib)
    monkeypatch.setattr(hostmem, "PINNED_MIN_BYTES", 1 << 16)
    monkeypatch.setattr(hostmem, "HELD_MAX", 8 << 20)
    monkeypatch.setattr(hostmem, "WAIT_MAX", 2 << 20)
    monkeypatch.setattr(hostmem, "_waiting", [])
    monkeypatch.setattr(hostmem, "_held", 0)
    yield lib
    gc.collect()


def test_bounds(pool):
    arrays = [hostmem.Result(n, 1 << 10).array for n in range(8, 520, 8)]  # 64 KB .. 4 MB
    assert pool.locked() == hostmem.held() <= 8 << 20
    for i, a in enumerate(arrays):
        a[...] = i
    assert all((a == i).all() for i, a in enumerate(arrays))
    del arrays, a
    assert pool.locked() == hostmem.held() <= 2 << 20
    hostmem.release()
    assert pool.locked() == hostmem.held() == 0


def test_reuse_and_views(pool):
    a = hostmem.Result(1 << 16).array
    at = a.ctypes.data
    view = a[5::7]
    del a
    b = hostmem.Result(1 << 16).array
    assert b.ctypes.data != at  # (the view keeps the block)
    del view
    c = hostmem.Result((1 << 16) - 99).array
    assert c.ctypes.data == at
    del b, c


class CollectingList(list):
    """Runs the garbage collector where it may run anyway: between a look at the list and its use."""

    def pop(self, *a):
        gc.collect()
        return list.pop(self, *a)


def test_collector_inside_the_pool(pool, monkeypatch):
    """Results in reference cycles are given back by a collector that runs inside the pool's code:
    every block keeps one user, and its size."""
    monkeypatch.setattr(hostmem, "_waiting", CollectingList())
    rng = numpy.random.default_rng(0)
    keep = []
    for i in range(40):
        gc.disable()
        for _ in range(3):
            cycle = [hostmem.Result(int(rng.integers(1 << 13, 1 << 16))).array]
            cycle.append(cycle)
        del cycle
        a = hostmem.Result(int(rng.integers(1 << 13, 1 << 16))).array
        gc.enable()
        a[...] = i
        keep.append((a, i))
        if len(keep) > 6:
            keep.pop(0)
        assert all((v == k).all() for v, k in keep)
        spans = sorted((v.ctypes.data, v.nbytes) for v, _ in keep)
        assert all(p + n <= q for (p, n), (q, _) in zip(spans, spans[1:]))
    del keep, a
    gc.collect()
    assert pool.locked() == hostmem.held() <= 2 << 20


def test_threads(pool):
    bad = []

    def work(i):
        rng = numpy.random.default_rng(i)
        for _ in range(300):
            a = hostmem.Result(int(rng.integers(1 << 13, 1 << 16))).array
            a[...] = i
            if not (a == i).all():
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    assert pool.locked() == hostmem.held() <= 2 << 20
