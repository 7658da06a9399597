"""MO coefficients of a spherical basis to and from its Cartesian rows (okg_fold_coeff,
okg_unfold_coeff) against products with the dense transform."""
import numpy
import pytest

from helpers import assert_fp64_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natom,nmo", [(2, 1), (7, 33), (40, 70)])
def test_fold_and_unfold_coefficients(natom, nmo):
    """The fold bit for bit (the same products in the same order), the unfold at the FP64 bar."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orbkit_gb300 import _lib, build, synthetic
    build.build()
    from orbkit_gb300.basis import DeviceBasis
    rng = numpy.random.default_rng(natom)
    geo = synthetic.random_geometry(rng, natom, 30.0)
    spec = synthetic.build_basis(rng, ["C"] * natom, with_f=True, spherical=True)
    b = DeviceBasis(geo, spec, torch.device("cuda", torch.cuda.current_device()))
    C = torch.as_tensor(rng.standard_normal((nmo, b.nao)), device="cuda")
    T = torch.as_tensor(b.T, device="cuda")
    dense = torch.empty((nmo, b.ncart), dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().okg_mo_from_ao(nmo, b.nao, _lib.ptr(C), _lib.ptr(T), b.ncart, b.ncart, _lib.ptr(dense),
                                          b.ncart, _lib.stream_handle()))
    assert torch.equal(b.c_eff(C), dense)
    G = torch.as_tensor(rng.standard_normal((nmo, b.ncart)), device="cuda")
    assert_fp64_close(b.c_grad(G).cpu().numpy(), (G @ T.T).cpu().numpy(), "unfold")
