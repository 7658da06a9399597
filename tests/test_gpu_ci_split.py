"""The detCI quadratic forms on the tensor cores: MO counts and point counts at the edges of
their tiles, against numpy in long double; non-finite MO values and coefficients."""
import numpy
import pytest

from helpers import assert_fp64_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def detci():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orbkit_gb300 import build
    build.build()
    from orbkit_gb300 import detci as d
    return d


def terms(rng, nmo, n):
    return [[[float(v)] for v in rng.standard_normal(n)], [[int(k)] for k in rng.integers(0, nmo, n)]], \
        [[float(v) for v in rng.standard_normal(3 * n)], [[int(a), int(b)] for a, b in rng.integers(0, nmo, (3 * n, 2))]]


def exact(zero, sing, mo, drv):
    ld = numpy.longdouble
    nmo = mo.shape[0]
    M, F = numpy.zeros((nmo, nmo), dtype=ld), numpy.zeros((nmo, nmo), dtype=ld)
    for c, k in zip(*zero):
        M[k[0], k[0]] += ld(c[0])
    for c, (a, b) in zip(*sing):
        M[a, b] += ld(c)
        F[a, b] += ld(c)
    mo, drv = mo.astype(ld), drv.astype(ld)
    t = (F - F.T).T @ mo
    return ((M @ mo) * mo).sum(0), -(t[None] * drv).sum(1) / 2


@pytest.mark.parametrize("nmo,npts", [(1, 1), (2, 129), (16, 128), (17, 1000), (32, 127), (33, 4097), (48, 20001), (64, 300),
                                      (65, 300)])
def test_against_long_double(detci, nmo, npts):
    rng = numpy.random.default_rng(nmo)
    zero, sing = terms(rng, nmo, 40)
    mo = rng.standard_normal((nmo, npts)) * numpy.exp(rng.uniform(-20, 2, npts))
    drv = rng.standard_normal((3, nmo, npts))
    r, j = exact(zero, sing, mo, drv)
    assert_fp64_close(detci.rho(zero, sing, mo, reference_slicing=False), r.astype(numpy.float64), "rho")
    assert_fp64_close(detci.jab(zero, sing, mo, drv, reference_slicing=False), j.astype(numpy.float64), "jab")


def test_non_finite_values(detci):
    """NaN at the points (and in every point, for a coefficient) where the sum has it."""
    rng = numpy.random.default_rng(5)
    zero, sing = terms(rng, 20, 200)
    mo, drv = rng.standard_normal((20, 700)), rng.standard_normal((3, 20, 700))
    clean = detci.rho(zero, sing, mo, reference_slicing=False)
    mo[3, 17] = numpy.nan
    mo[:, 500] = 0.0
    r = detci.rho(zero, sing, mo, reference_slicing=False)
    assert numpy.isnan(r[17]) and r[500] == 0.0
    keep = [i for i in range(700) if i not in (17, 500)]
    assert (r[keep] == clean[keep]).all()
    sing[0][0] = numpy.nan
    assert numpy.isnan(detci.rho(zero, sing, mo, reference_slicing=False)).sum() >= 698
    assert numpy.isnan(detci.jab(zero, sing, mo, drv, reference_slicing=False)).all()
