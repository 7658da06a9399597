"""Expired waits in the tensor-core FP64 kernels, without a GPU fault: every wait is bounded,
and with a limit of one poll, or none, the waits run out on purpose.  The outputs of such a call are
still complete, and are the bits of the general kernels that compute it then; the next call
has the usual bits again; calls of other host threads keep the usual limit.
"""
import ctypes
import threading

import numpy
import pytest

from test_gpu_split64_range import device_call, molecule, near_points

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


class limited:
    """Waits of one poll (or none) in the calling thread."""

    def __init__(self, polls):
        self.polls = polls

    def __enter__(self):
        from orbkit_gb300 import _lib
        _lib.check(_lib.load().okg_set_wait_limit(self.polls))

    def __exit__(self, *exc):
        from orbkit_gb300 import _lib
        _lib.check(_lib.load().okg_set_wait_limit(1 << 24))


def captured(run):
    """The call in a graph: the general kernel."""
    import torch
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    graph.replay()
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("what,codes", [("rho", []), ("rho", [1, 2, 3]), ("rho", [4, 5, 6]), ("mo", [0]), ("mo", [2]), ("mo", [6])])
def test_density_and_orbitals(core, what, codes):
    import torch
    from orbkit_gb300 import _lib
    L = _lib.load()
    qc = molecule("f", nmo=40)
    b, C, occ, xyz, gd, n = device_call(core, qc, near_points(qc, 20001))

    def run():
        out = [torch.zeros((max(1, len(codes)) * (40 if what == "mo" else 1), n), dtype=torch.float64, device=C.device)]
        cc = _lib.int_array(codes)
        if what == "mo":
            _lib.check(L.okg_eval_mo(b.handle, gd, 40, _lib.ptr(C), len(codes), cc, 0, _lib.ptr(out[0]), n, _lib.stream_handle()))
        else:
            out.append(torch.zeros(n, dtype=torch.float64, device=C.device))
            _lib.check(L.okg_rho(b.handle, gd, 40, _lib.ptr(C), _lib.ptr(occ), len(codes), cc, 0, _lib.ptr(out[1]),
                                 _lib.ptr(out[0]), n, None, _lib.stream_handle()))
        return out

    usual = run()
    general = captured(run)
    assert not all(torch.equal(u, g) for u, g in zip(usual, general))  # (the two kernels round differently)
    other = []
    for polls in (1, 0, 1):
        with limited(polls):
            got = run()
            t = threading.Thread(target=lambda: other.append(run()))
            t.start()
            t.join()
        again = run()
        torch.cuda.synchronize()
        for o, g, a, u, t in zip(got, general, again, usual, other[-1]):
            assert torch.equal(o, g) and torch.equal(a, u) and torch.equal(t, u)


@pytest.mark.parametrize("precision", [64, 32])
def test_adjoint(core, precision):
    import torch
    from orbkit_gb300 import _lib, adjoint
    L = adjoint._L()
    qc = molecule("f", nmo=40)
    b, C, occ, xyz, gd, n = device_call(core, qc, near_points(qc, 20001))
    gen = torch.Generator(device=C.device).manual_seed(5)
    g = torch.randn((4, n), generator=gen, dtype=torch.float64, device=C.device)
    size = ctypes.c_size_t(0)
    _lib.check(L.okg_rho_backward_workspace(b.handle, gd, 40, precision, ctypes.byref(size)))

    def run(nbytes=size.value):
        work = torch.full((nbytes,), 255, dtype=torch.uint8, device=C.device)
        out = [torch.empty(s, dtype=torch.float64, device=C.device) for s in (tuple(C.shape), (b.nprim, 2), (b.natom, 3))]
        _lib.check(L.okg_rho_backward(b.handle, gd, 40, _lib.ptr(C), _lib.ptr(occ), _lib.ptr(g[0]), _lib.ptr(g[1]), n, precision,
                                      *[_lib.ptr(o) for o in out], _lib.ptr(work), nbytes, _lib.stream_handle()))
        return out

    usual, general = run(), run(size.value - 256)  # (that workspace fits the one-kernel form alone)
    assert not torch.equal(usual[0], general[0])
    for polls in (1, 0, 1):
        with limited(polls):
            got = run()
        again = run()
        torch.cuda.synchronize()
        for o, v, a, u in zip(got, general, again, usual):
            assert torch.equal(o, v) and torch.equal(a, u)


def ci_run(nmo, npts, flux, seed=0, change=None, pad=0):
    """okg_ci_rho_matrix / okg_ci_flux_matrix; pad: MOs of zeros appended (above 64 MOs the general
    kernel runs, its sums unchanged)."""
    import torch
    from orbkit_gb300 import _lib, detci
    L = detci._L()
    rng = numpy.random.default_rng(seed)
    mo, drv = rng.standard_normal((nmo, npts)), rng.standard_normal((3, nmo, npts))
    q = rng.standard_normal((nmo, nmo))
    if not flux:
        q = numpy.tril(q)
    if change:
        change(mo, drv, q)
    m = nmo + pad
    qt = numpy.zeros((m, (m + 15) // 16 * 16))
    qt[:nmo, :nmo] = q
    mo = numpy.concatenate([mo, numpy.zeros((pad, npts))])
    drv = numpy.concatenate([drv, numpy.zeros((3, pad, npts))], axis=1)
    mo, drv, qt = (torch.as_tensor(numpy.ascontiguousarray(v), device="cuda") for v in (mo, drv, qt))
    out = torch.zeros((3 if flux else 1, npts), dtype=torch.float64, device="cuda")
    if flux:
        _lib.check(L.okg_ci_flux_matrix(npts, _lib.ptr(mo), _lib.ptr(drv), npts, m, _lib.ptr(qt), -0.5, _lib.ptr(out),
                                        _lib.stream_handle()))
    else:
        _lib.check(L.okg_ci_rho_matrix(npts, _lib.ptr(mo), npts, m, _lib.ptr(qt), _lib.ptr(out), _lib.stream_handle()))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("flux", [False, True])
@pytest.mark.parametrize("nmo", [1, 24, 42, 64])
def test_detci(core, nmo, flux):
    npts = 50003
    usual, general = ci_run(nmo, npts, flux), ci_run(nmo, npts, flux, pad=65 - nmo)
    for polls in (1, 0, 1):
        with limited(polls):
            got = ci_run(nmo, npts, flux)
        # (with one poll some blocks are done in time and have the usual bits)
        assert ((got == general) | (got == usual)).all()
        assert polls or numpy.array_equal(got, general)
        assert numpy.array_equal(ci_run(nmo, npts, flux), usual)


def _mo(i, p, v):
    return lambda mo, drv, q: mo.__setitem__((i, p), v)


@pytest.mark.parametrize("flux", [False, True])
@pytest.mark.parametrize("change", [_mo(3, 200, numpy.inf), _mo(3, 200, numpy.nan), _mo(3, slice(None), -numpy.inf), _mo(0, 5000, 1e305),
                                    lambda mo, drv, q: q.__setitem__((5, 2), numpy.inf), lambda mo, drv, q: q.__setitem__((5, 2), numpy.nan),
                                    lambda mo, drv, q: q.__imul__(1e-280)])
def test_detci_beyond_the_digits(core, change, flux):
    """Infinities, NaN and sizes that the digits cannot hold: what the general kernel gives."""
    with numpy.errstate(all="ignore"):
        a, b = ci_run(20, 5003, flux, change=change), ci_run(20, 5003, flux, change=change, pad=45)
        assert ((a == b) | (numpy.isnan(a) & numpy.isnan(b)) | (numpy.abs(a - b) <= 1e-12 * numpy.abs(b[numpy.isfinite(b)]).max(initial=0.0))).all()


def test_wait_limit_argument_checked(core):
    from orbkit_gb300 import _lib
    with pytest.raises(_lib.OkgError):
        _lib.check(_lib.load().okg_set_wait_limit(-1))


@pytest.mark.parametrize("flux", [False, True])
@pytest.mark.parametrize("nmo", [20, 42])
@pytest.mark.parametrize("last", [False, True])
def test_detci_points_beyond_the_digits(core, nmo, flux, last):
    """Such points in any of a block's tiles, or in the last one alone: they have the general
    kernel's bits, the others the usual ones."""
    npts = 150007
    at = numpy.array([npts - 1]) if last else numpy.concatenate([numpy.arange(0, npts, 997), numpy.arange(70000, 70128)])

    def change(mo, drv, q):
        mo[nmo // 2, at] = numpy.where(at % 2 == 0, numpy.inf, -1e305)

    got, general, usual = (ci_run(nmo, npts, flux, change=c, pad=p) for c, p in ((change, 0), (change, 65 - nmo), (None, 0)))
    beyond = numpy.zeros(npts, dtype=bool)
    beyond[at] = True
    assert numpy.array_equal(got[:, beyond], general[:, beyond], equal_nan=True)
    assert numpy.array_equal(got[:, ~beyond], usual[:, ~beyond])
