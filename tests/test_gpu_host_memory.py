"""Page-locked results: bounded, given back, never shared, the same values with and without."""
import gc
import threading

import numpy
import pytest

from test_gpu_split64_range import molecule

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orbkit_gb300 import build
    build.build()
    from orbkit_gb300 import core as c
    c.quiet = True
    return c


def orbitals(core, qc, n, shift=0.0):
    axes = [numpy.linspace(-3.0 + shift, 3.0, k) for k in (n, 16, 16)]
    return core.rho_compute_no_slice(qc, calc_mo=True, x=axes[0], y=axes[1], z=axes[2], is_vector=False)


def test_bounded_and_never_shared(core, monkeypatch):
    """40 results of about 1 MB in the caller's hands with 8 MB to lock and 2 MB to keep waiting."""
    from orbkit_gb300 import hostmem
    gc.collect()
    hostmem.release()
    base = hostmem.held()
    monkeypatch.setattr(hostmem, "HELD_MAX", base + (8 << 20))
    monkeypatch.setattr(hostmem, "WAIT_MAX", 2 << 20)
    qc = molecule("p")
    results = []
    for i in range(40):
        results.append(orbitals(core, qc, 64 + i % 3, 0.01 * i))
        assert hostmem.held() <= base + (8 << 20)
    assert hostmem.held() > base
    monkeypatch.setattr(hostmem, "PINNED_MIN_BYTES", 1 << 60)
    for i, r in enumerate(results):
        assert numpy.array_equal(r, orbitals(core, qc, 64 + i % 3, 0.01 * i))
    del results, r
    gc.collect()
    assert hostmem.held() <= base + (2 << 20)
    hostmem.release()
    assert hostmem.held() == base


def test_views_keep_the_block(core):
    qc = molecule("p")
    view = orbitals(core, qc, 80)[2, ::3]
    want = view.copy()
    for i in range(5):
        orbitals(core, qc, 80, 0.1 * i)
    assert numpy.array_equal(view, want)


def test_locking_fails(core, monkeypatch):
    """The host refuses to lock pages: an ordinary array."""
    from orbkit_gb300 import _lib, hostmem
    qc = molecule("p")
    want = orbitals(core, qc, 128)
    hostmem.release()

    class Refusing:
        def okg_host_alloc(self, size, p):
            return -4

        def __getattr__(self, name):
            return getattr(_lib._lib, name)

    monkeypatch.setattr(hostmem._lib, "load", lambda: Refusing())
    got = orbitals(core, qc, 128)
    monkeypatch.undo()
    assert got.flags.owndata or got.base.flags.owndata
    assert numpy.array_equal(got, want)


@pytest.mark.parametrize("limit", [1 << 16, 1 << 20])
def test_results_in_slices(core, monkeypatch, limit):
    """Results read back in several ranges of points."""
    qc = molecule("d")
    axes = [numpy.linspace(-3.0, 3.0, k) for k in (30, 25, 23)]
    core.grid.set_grid(*axes, is_vector=False)
    ao = core.ao_creator(qc.geo_spec, qc.ao_spec)

    def all_results():
        return [core.ao_creator(qc.geo_spec, qc.ao_spec, drv="x"), core.mo_creator(ao, qc.mo_spec), core.calc_mo_matrix(qc),
                core.rho_compute(qc, calc_mo=True)]

    want = all_results()
    monkeypatch.setattr(core, "MAX_SLICE_BYTES", limit)
    for a, b in zip(all_results(), want):
        assert a.shape == b.shape and (numpy.abs(a - b) <= 1e-12 * numpy.abs(b).max()).all()


def test_threads(core):
    """Results of several host threads at once."""
    import torch
    qc = molecule("p")
    want = [orbitals(core, qc, 100 + i) for i in range(4)]
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                if not numpy.array_equal(orbitals(core, qc, 100 + i), want[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_evaluation_that_raises(core, monkeypatch):
    """A block whose evaluation raised after a part was queued is complete before it is used again."""
    from orbkit_gb300 import _lib, hostmem
    qc = molecule("d")
    axes = [numpy.linspace(-3.0, 3.0, k) for k in (64, 32, 32)]
    want = orbitals(core, qc, 128)
    real, calls = hostmem.Result.put, []

    def put(self, i, j, part):
        real(self, i, j, part)
        calls.append(self)
        raise _lib.OkgError(-1, "on purpose")

    monkeypatch.setattr(hostmem.Result, "put", put)
    with pytest.raises(_lib.OkgError):
        core.rho_compute_no_slice(qc, calc_mo=True, x=axes[0], y=axes[1], z=axes[2], is_vector=False)
    assert len(calls) == 1
    calls.clear()
    monkeypatch.undo()
    gc.collect()
    assert numpy.array_equal(orbitals(core, qc, 128), want)


@pytest.mark.parametrize("thread", [False, True])
def test_while_a_graph_is_captured(core, thread):
    """Blocks locked and freed while a stream is captured (a result made by another thread, results
    that the collector drops): the capture holds, and the results stay page-locked."""
    import torch
    from orbkit_gb300 import hostmem
    x = torch.arange(1024.0, device="cuda")
    torch.cuda.synchronize()
    addresses = []

    def work():
        r = hostmem.Result(1 << 17)
        addresses.append(r.address)
        r.array[:] = 1.0
        del r
        hostmem.release()

    gc.collect()
    hostmem.release()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = x * 2.0
        if thread:
            t = threading.Thread(target=work)
            t.start()
            t.join()
        else:
            work()
        z = y + 1.0
    assert addresses[0] is not None
    x.fill_(3.0)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((z == 7.0).all())
