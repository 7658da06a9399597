"""The tensor-core FP64 path where a tile of points, a parameter or a coefficient leaves the
ordinary range: the same values as the DFMA kernel (the same points in small calls).

Bar at every point: 1e-12 of the sum of the magnitudes of what is added there, taken from
the AOs (the rounding of an FP64 sum of a few hundred terms is below 1e-13 of it); of a
derivative, the largest of its three directions.
"""
import numpy
import pytest

pytestmark = pytest.mark.gpu
RTOL = 1e-12


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


def molecule(top, nmo=7, seed=1):
    """Four atoms; per atom a steep s contraction (exponents to 1e7) and a shell of every type
    up to `top`; dense coefficients."""
    from orbkit_gb300 import synthetic
    from orbkit_gb300.orbitals import AOClass, MOClass
    rng = numpy.random.default_rng(seed)
    geo = rng.uniform(-3.0, 3.0, (4, 3))
    ao = [{"atom": a, "type": "s", "pnum": 8, "coeffs": numpy.stack([10.0 ** numpy.arange(7.0, -1.0, -1.0),
                                                                    rng.uniform(0.5, 1.0, 8)], axis=1)} for a in range(4)]
    for a in range(4):
        for lt in "spdfg"[:"spdfg".index(top) + 1]:
            ao.append({"atom": a, "type": lt, "pnum": 2,
                       "coeffs": numpy.stack([rng.uniform(0.1, 30.0, 2), rng.uniform(0.5, 1.0, 2)], axis=1)})
    spec = AOClass(ao)
    spec.update()
    C = rng.uniform(0.5, 1.0, (nmo, spec.get_ao_num())) * rng.choice([-1.0, 1.0], (nmo, spec.get_ao_num()))
    mo = MOClass([{"coeffs": C[i], "occ_num": 1.0 + i % 2, "energy": 0.0, "sym": "%d.1" % (i + 1)} for i in range(nmo)])
    mo.update()
    return synthetic.make_qc(geo, ["C"] * 4, spec, mo)


KW = {"rho": {}, "grad": {"drv": ["x", "y", "z"]}, "laplacian": {"laplacian": True}, "mo": {"calc_mo": True}}


def call(core, qc, what, pts):
    out = core.rho_compute_no_slice(qc, x=pts[0], y=pts[1], z=pts[2], is_vector=True, **KW[what])
    return list(out) if isinstance(out, tuple) else [out]


def sums(core, qc, what, pts):
    """Per output (laplacian: density, its three second derivatives, their sum), the sum of
    magnitudes at every point."""
    C, occ = numpy.abs(qc.mo_spec.get_coeffs()), numpy.abs(qc.mo_spec.get_occ())[:, None]
    mag = lambda drv: C @ numpy.abs(core.ao_creator(qc.geo_spec, qc.ao_spec, drv=drv, x=pts[0], y=pts[1], z=pts[2], is_vector=True))
    m0 = mag(None)
    if what == "mo":
        return [m0]
    rho = (occ * m0 * m0).sum(0)
    if what == "rho":
        return [rho]
    first = numpy.max([mag(d) for d in "xyz"], axis=0)
    if what == "grad":
        return [rho, (2.0 * occ * m0 * first).sum(0)]
    second = (2.0 * occ * (m0 * numpy.max([mag(d + d) for d in "xyz"], axis=0) + first * first)).sum(0)
    return [rho, second, 3.0 * second]


def both_routes(core, qc, what, pts):
    """The call whole (tensor cores) and in runs of 300 points (DFMA kernel)."""
    whole = call(core, qc, what, pts)
    runs = [call(core, qc, what, pts[:, i:i + 300]) for i in range(0, pts.shape[1], 300)]
    return whole, [numpy.concatenate([r[k] for r in runs], axis=-1) for k in range(len(whole))]


def compare(core, qc, what, pts):
    a, b = both_routes(core, qc, what, pts)
    for u, v, s in zip(a, b, sums(core, qc, what, pts)):
        assert numpy.array_equal(numpy.isnan(u), numpy.isnan(v))
        bad = ~(numpy.abs(u - v) <= RTOL * s) & ~numpy.isnan(v)
        assert not bad.any(), "%s: %d of %d" % (what, bad.sum(), bad.size)


def near_points(qc, n, seed=2):
    """Points at 1e-4 .. 1 bohr from the nuclei."""
    rng = numpy.random.default_rng(seed)
    d = rng.standard_normal((n, 3))
    d *= (10.0 ** rng.uniform(-4.0, 0.0, n) / numpy.linalg.norm(d, axis=1))[:, None]
    return (qc.geo_spec[rng.integers(0, len(qc.geo_spec), n)] + d).T.copy()


@pytest.mark.parametrize("what", ["rho", "grad", "laplacian", "mo"])
@pytest.mark.parametrize("top", ["s", "d"])
@pytest.mark.parametrize("far", [1e3, 1e5, 1e7, 1e8])
def test_tiles_led_by_a_far_point(core, what, top, far):
    """The first point of every tile (32 and 128 points) far from all atoms, the others near
    nuclei: coordinates relative to the first have no digits left for the distances."""
    qc = molecule(top)
    pts = near_points(qc, 6016)
    pts[0, ::32] = far
    pts[1, ::64] = -far
    compare(core, qc, what, pts)
