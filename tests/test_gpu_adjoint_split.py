"""The tensor-core adjoint (okg_adjoint_split.cu, up to 64 MOs) at the edges of its tiles,
digit panels and runs, against a float64 PyTorch reference gradient.

Bars, normwise relative per parameter block: FP64 1e-10 and FP32 2e-3, those of the
one-kernel form (sums of a few thousand terms of relative error 1e-14 and 1e-6 with
cancellation of up to 1e3).
"""
import ctypes

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from orbkit_gb300 import build
    build.build()
    return t


def molecule(nmo, seed, natom=4, top="f", spherical=False):
    """Shells of every type up to `top`, 1 to 11 primitives."""
    from orbkit_gb300 import synthetic
    from orbkit_gb300.orbitals import AOClass, MOClass
    rng = numpy.random.default_rng(seed)
    geo = synthetic.random_geometry(rng, natom, 5.0)
    ao = []
    for a in range(natom):
        for lt in "spdfg"[:"spdfg".index(top) + 1]:
            for n in ((11, 1) if lt == "s" else (3,)):
                alpha = numpy.exp(rng.uniform(numpy.log(0.1), numpy.log(2e3 if lt == "s" else 10.0), n))
                ao.append({"atom": a, "type": lt, "pnum": n,
                           "coeffs": numpy.stack([alpha, rng.uniform(-1.0, 1.0, n)], axis=1)})
    spec = AOClass(ao)
    if spherical:
        spec.set_lm_dict(p=[1, 0])
    spec.update()
    C = rng.uniform(-1.0, 1.0, (nmo, spec.get_ao_num()))
    mo = MOClass([{"coeffs": C[i], "occ_num": float(rng.uniform(0.1, 2.0)), "energy": 0.0, "sym": "%d.1" % (i + 1)}
                  for i in range(nmo)])
    mo.update()
    return synthetic.make_qc(geo, ["C"] * natom, spec, mo), rng


def params(torch, qc):
    prim = qc.ao_spec.get_prim_coeffs()
    return [torch.tensor(numpy.array(v), dtype=torch.float64, device="cuda", requires_grad=True)
            for v in (qc.mo_spec.get_coeffs(), prim[:, 0], prim[:, 1], qc.geo_spec)]


CASES = [(nmo, npts, top, sph) for nmo, npts, top, sph in
         ((1, 1, "p", False), (2, 31, "g", False), (15, 33, "d", False), (16, 127, "d", True), (17, 128, "f", False),
          (32, 129, "f", True), (33, 257, "p", False), (48, 1000, "g", False), (49, 640, "d", True), (63, 2049, "f", False),
          (64, 4097, "d", False), (65, 300, "d", False))]


@pytest.mark.parametrize("prec,bar", [("fp64", 1e-10), ("fp32", 2e-3)])
@pytest.mark.parametrize("nmo,npts,top,spherical", CASES)
def test_against_float64_reference(torch, nmo, npts, top, spherical, prec, bar):
    import torch_ref
    from orbkit_gb300.adjoint import DensityModel
    qc, rng = molecule(nmo, nmo, top=top, spherical=spherical)
    npts += 2047 if prec == "fp32" else 0  # (2048 points on; fewer are the one-kernel form's)
    pts = rng.uniform(-3.0, 3.0, (3, npts))
    pts[:, 0] = qc.geo_spec[1]  # a nucleus
    model = DensityModel(qc, pts[0], pts[1], pts[2], True, prec)
    u = torch.tensor(rng.uniform(-1, 1, npts), device="cuda")
    v = torch.tensor(rng.uniform(-1, 1, (3, npts)), device="cuda")
    got, ref = params(torch, qc), params(torch, qc)
    rho, grad = model(*got)
    ((u * rho).sum() + (v * grad).sum()).backward()
    st = torch_ref.Structure(qc.ao_spec, model.basis.T)
    r, g = torch_ref.rho_grad(*ref, st, model.occ, torch.tensor(pts, device="cuda"))
    ((u * r).sum() + (v * g).sum()).backward()
    for name, a, b in zip(("C", "alpha", "c", "R"), got, ref):
        err = float((a.grad - b.grad).abs().max() / b.grad.abs().max())
        assert err <= bar, (name, err)


def backward(torch, model, par, g_rho, g_grad, short=False):
    """okg_rho_backward; `short`: a workspace that only the one-kernel form fits in."""
    from orbkit_gb300 import _lib
    C = model.basis.c_eff(par[0].detach())
    need = ctypes.c_size_t(0)
    prec = 64 if model.precision == "fp64" else 32
    _lib.check(model._L.okg_rho_backward_workspace(model.basis.handle, model.gd, model.nmo, prec, ctypes.byref(need)))
    work = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out = [torch.empty_like(C), torch.empty((model.basis.nprim, 2), dtype=torch.float64, device="cuda"),
           torch.empty((model.basis.natom, 3), dtype=torch.float64, device="cuda")]
    _lib.check(model._L.okg_rho_backward(model.basis.handle, model.gd, model.nmo, _lib.ptr(C), _lib.ptr(model.occ),
                                         _lib.ptr(g_rho), _lib.ptr(g_grad) if g_grad is not None else None, model.npts, prec,
                                         *(_lib.ptr(o) for o in out), _lib.ptr(work), need.value - (1 if short else 0),
                                         _lib.stream_handle()))
    return out


@pytest.mark.parametrize("prec,bar", [("fp64", 1e-10), ("fp32", 2e-3)])
@pytest.mark.parametrize("what", ["grid", "no_gradient", "runs"])
def test_against_one_kernel_form(torch, what, prec, bar):
    """Regular grids (odd edges), densities alone, and more points than one run holds."""
    from orbkit_gb300.adjoint import DensityModel
    qc, rng = molecule(60 if what == "runs" else 19, 5, natom=6, top="d")
    n = (131, 119, 121) if what == "runs" else (23, 37, 41)
    axes = [numpy.linspace(-4.0, 4.0, k) for k in n]
    model = DensityModel(qc, *axes, False, prec)
    par = params(torch, qc)
    model._set(*(p.detach() for p in par[1:]))
    u = torch.tensor(rng.uniform(-1, 1, model.npts), device="cuda")
    v = None if what == "no_gradient" else torch.tensor(rng.uniform(-1, 1, (3, model.npts)), device="cuda")
    for a, b in zip(backward(torch, model, par, u, v), backward(torch, model, par, u, v, short=True)):
        assert float((a - b).abs().max() / b.abs().max()) <= bar
        assert bool(torch.isfinite(a).all())


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_cotangent_not_a_number(torch, prec):
    """One cotangent that is not a number reaches every derivative that its point enters."""
    from orbkit_gb300.adjoint import DensityModel
    qc, rng = molecule(9, 7, top="d")
    pts = rng.uniform(-3.0, 3.0, (3, 20000))
    model = DensityModel(qc, pts[0], pts[1], pts[2], True, prec)
    par = params(torch, qc)
    model._set(*(p.detach() for p in par[1:]))
    u = torch.ones(20000, dtype=torch.float64, device="cuda")
    u[777] = float("nan")
    v = torch.zeros((3, 20000), dtype=torch.float64, device="cuda")
    for short in (False, True):
        for o in backward(torch, model, par, u, v, short):
            assert bool(torch.isnan(o).all()), short
