"""Calls of several host threads with different shared-memory sizes of the same kernels: every
launch succeeds and has the bits of the call alone."""
import ctypes
import threading

import numpy
import pytest

from test_gpu_split64_range import device_call, molecule, near_points

pytestmark = pytest.mark.gpu
CALLS = 5000


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


def density(core, nmo):
    import torch
    from orbkit_gb300 import _lib
    L = _lib.load()
    qc = molecule("s", nmo=nmo)
    b, C, occ, xyz, gd, n = device_call(core, qc, near_points(qc, 4900))
    rho = torch.empty(n, dtype=torch.float64, device=C.device)
    return lambda keep=(b, xyz): L.okg_rho(b.handle, gd, nmo, _lib.ptr(C), _lib.ptr(occ), 0, _lib.int_array([]), 0, _lib.ptr(rho), None,
                                           n, None, _lib.stream_handle()), rho


def backward(core, nmo):
    import torch
    from orbkit_gb300 import _lib, adjoint
    L = adjoint._L()
    qc = molecule("s", nmo=nmo)
    b, C, occ, xyz, gd, n = device_call(core, qc, near_points(qc, 200))
    g = torch.ones((4, n), dtype=torch.float64, device=C.device)
    size = ctypes.c_size_t(0)
    _lib.check(L.okg_rho_backward_workspace(b.handle, gd, nmo, 64, ctypes.byref(size)))
    work = torch.empty(size.value, dtype=torch.uint8, device=C.device)
    out = [torch.empty(s, dtype=torch.float64, device=C.device) for s in (tuple(C.shape), (b.nprim, 2), (b.natom, 3))]
    return lambda keep=(b, xyz, work): L.okg_rho_backward(
        b.handle, gd, nmo, _lib.ptr(C), _lib.ptr(occ), _lib.ptr(g[0]), _lib.ptr(g[1]), n, 64, *[_lib.ptr(o) for o in out],
        _lib.ptr(work), size.value, _lib.stream_handle()), out[0]


def detci(core, nmo):
    import torch
    from orbkit_gb300 import _lib, detci as d
    L = d._L()
    mo = torch.randn((nmo, 300), dtype=torch.float64, device="cuda")
    q = torch.randn((nmo, (nmo + 15) // 16 * 16), dtype=torch.float64, device="cuda").tril()
    q[:, nmo:] = 0
    out = torch.empty(300, dtype=torch.float64, device="cuda")
    return lambda keep=(mo, q): L.okg_ci_rho_matrix(300, _lib.ptr(mo), 300, nmo, _lib.ptr(q), _lib.ptr(out), _lib.stream_handle()), out


@pytest.mark.parametrize("make,sizes", [(density, (5, 40)), (backward, (5, 60)), (detci, (8, 30)), (detci, (40, 64))])
def test_sizes_in_turn(core, make, sizes):
    import torch
    calls = [make(core, n) for n in sizes]
    want = []
    for run, out in calls:
        assert run() == 0
        torch.cuda.synchronize()
        want.append(out.clone())
    status = [[], []]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(CALLS):
                status[i].append(calls[i][0]())
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not any(any(s) for s in status), [len([v for v in s if v]) for s in status]
    for (run, out), w in zip(calls, want):
        assert torch.equal(out, w)
