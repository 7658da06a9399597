"""Workspace of the adjoint: bounded whatever the number of points."""
import ctypes

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


def workspace(b, gd, nmo, precision):
    from orbkit_gb300 import _lib, adjoint
    size = ctypes.c_size_t(0)
    _lib.check(adjoint._L().okg_rho_backward_workspace(b.handle, gd, nmo, precision, ctypes.byref(size)))
    return size.value


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nmo", [5, 64])
def test_does_not_grow_with_the_points(core, nmo, precision):
    qc = molecule("g")
    b, C, occ, xyz, gd, n = device_call(core, qc, near_points(qc, 8))
    for npts in (1 << 22, 1 << 24, 1 << 27):
        gd.npts = npts
        assert workspace(b, gd, nmo, precision) <= 1.25 * 2 ** 30


@pytest.mark.parametrize("precision", [64, 32])
def test_bases_beyond_the_tables(core, precision):
    """More shells than the tensor-core kernels' tables hold: the one-kernel form's workspace
    (that of 65 MOs, but for the MOs)."""
    import torch
    from orbkit_gb300.orbitals import AOClass
    rng = numpy.random.default_rng(3)
    ao = AOClass([{"atom": i % 9, "type": "s", "pnum": 1, "coeffs": numpy.array([[rng.uniform(0.1, 9.0), 1.0]])} for i in range(2049)])
    ao.update()
    b = core.get_basis(rng.uniform(-3.0, 3.0, (9, 3)), ao, torch.device("cuda"))
    qc = molecule("s")
    _, _, _, xyz, gd, n = device_call(core, qc, near_points(qc, 6000))
    assert workspace(b, gd, 64, precision) <= workspace(b, gd, 65, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_device_without_room(core, precision, monkeypatch):
    """A fit step where the whole workspace cannot be allocated: the gradients of the form that
    needs the least, and those of the other again once there is room."""
    import torch
    from orbkit_gb300.adjoint import DensityModel
    qc = molecule("d", nmo=40)
    pts = near_points(qc, 20000)
    model = DensityModel(qc, pts[0], pts[1], pts[2], True, precision)
    prim = qc.ao_spec.get_prim_coeffs()
    par = [torch.tensor(numpy.array(v), dtype=torch.float64, device="cuda", requires_grad=True)
           for v in (qc.mo_spec.get_coeffs(), prim[:, 0], prim[:, 1], qc.geo_spec)]

    def step():
        for p in par:
            p.grad = None
        rho, grad = model(*par)
        (rho.sum() + (grad ** 2).sum()).backward()
        return [p.grad.clone() for p in par]

    usual = step()
    whole = model._work.numel()
    model._work = None
    empty = torch.empty

    def no_room(*a, **k):
        if a and a[0] == whole:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", no_room)
    least = step()
    assert model._work.numel() < whole
    monkeypatch.undo()
    again = step()
    assert model._work.numel() == whole
    bar = 1e-10 if precision == "fp64" else 2e-3  # (as in test_gpu_adjoint_split.py)
    for u, l, a in zip(usual, least, again):
        assert torch.equal(u, a)
        assert float((u - l).abs().max() / u.abs().max()) <= bar
