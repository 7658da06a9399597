"""The stated error of the tensor-core FP64 path, point by point: n 2^-50 max|C| max|AO| (of a
derivative, the largest in any direction), for orbitals whose coefficients reach over many
orders of magnitude.  (Per column of fixed-point digits 2^-53 2^E 2^F, with 2^F below 2.1 times
the largest coefficient and 2^E below 4 times the largest AO: its power of two, the margin of
the bound and the power of two of the angular norm.)"""
import numpy
import pytest

from test_gpu_split64_range import call, molecule

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


@pytest.mark.parametrize("outside", [0.0, 1e-14, 1e-7])
@pytest.mark.parametrize("top", ["p", "g"])
def test_localised_orbitals(core, top, outside):
    qc = molecule(top, nmo=12)
    atom = numpy.array([ao["atom"] for ao in qc.ao_spec])[qc.ao_spec.get_assign_lxlylz_to_cont()]
    for i in range(12):
        mo = qc.mo_spec[i]
        mo["coeffs"] = numpy.where(atom == i % 4, mo["coeffs"], outside * mo["coeffs"])
    qc.mo_spec.update()
    pts = numpy.random.default_rng(8).uniform(-4.0, 4.0, (3, 6000))
    pts[:, :4] = qc.geo_spec.T
    C = qc.mo_spec.get_coeffs()
    big = numpy.abs(C).max(1)[:, None]
    for drvs in ([None], ["x", "y", "z"], ["xx", "yy", "zz"]):
        ao = [core.ao_creator(qc.geo_spec, qc.ao_spec, drv=d, x=pts[0], y=pts[1], z=pts[2], is_vector=True) for d in drvs]
        top_ao = numpy.max([numpy.abs(a).max(0) for a in ao], axis=0)
        for d, a in zip(drvs, ao):
            got = core.rho_compute_no_slice(qc, calc_mo=True, drv=d, x=pts[0], y=pts[1], z=pts[2], is_vector=True)
            want = C.astype(numpy.longdouble) @ a
            got = got[0] if d else got
            # (the AOs themselves carry roundings of their own: 2^-48 sum |C| |AO|)
            bar = C.shape[1] * 2.0 ** -50 * big * top_ao + 2.0 ** -48 * (numpy.abs(C) @ numpy.abs(a))
            assert (numpy.abs(got - want) <= bar).all(), (d, float((numpy.abs(got - want) / bar).max()))


def test_densities_of_delocalised_orbitals(core):
    """Where every MO holds every AO the density is as accurate as an FP64 sum, point by point."""
    qc = molecule("g", nmo=12)
    pts = numpy.random.default_rng(9).uniform(-9.0, 9.0, (3, 6000))
    rho = call(core, qc, "rho", pts)[0]
    C, occ = qc.mo_spec.get_coeffs(), qc.mo_spec.get_occ()[:, None]
    a = core.ao_creator(qc.geo_spec, qc.ao_spec, x=pts[0], y=pts[1], z=pts[2], is_vector=True)
    mo = C.astype(numpy.longdouble) @ a
    size = (occ * (numpy.abs(C) @ numpy.abs(a)) ** 2).sum(0)
    assert (numpy.abs(rho - (occ * mo * mo).sum(0)) <= 1e-13 * size).all()
