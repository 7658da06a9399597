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
    with numpy.errstate(all="ignore"):
        for u, v, s in zip(a, b, sums(core, qc, what, pts)):
            bad = ~((u == v) | (numpy.isnan(u) & numpy.isnan(v)) | (numpy.abs(u - v) <= RTOL * s))
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


@pytest.mark.parametrize("what", ["rho", "grad", "laplacian", "mo"])
@pytest.mark.parametrize("top", ["s", "g"])
@pytest.mark.parametrize("far", [1e9, 1e12, 1e25, 1e60, 1e200, numpy.inf])
def test_points_beyond_every_atom(core, what, top, far):
    """Zero where every exponential is zero and its polynomial finite, else NaN."""
    qc = molecule(top)
    pts = near_points(qc, 6016)
    pts[2, 100] = -far
    pts[:, 3000] = far
    pts[1, 4096:4128] = far  # whole tiles of 32 points
    compare(core, qc, what, pts)


def edit(qc, alpha=None, scale=None, position=None, coeff=None, row=None):
    """One exponent, the contraction coefficients of one shell, one position, one MO
    coefficient or the size of one MO replaced."""
    if alpha is not None:
        qc.ao_spec[1]["coeffs"][3, 0] = alpha
    if scale is not None:
        qc.ao_spec[2]["coeffs"][:, 1] *= scale
    qc.ao_spec.update()
    if position is not None:
        qc.geo_spec[2, 1] = position
    if coeff is not None:
        qc.mo_spec[4]["coeffs"][2] = coeff
    if row is not None:
        qc.mo_spec[4]["coeffs"] = qc.mo_spec[4]["coeffs"] * row
    qc.mo_spec.update()
    return qc


OUTSIDE = [{"alpha": 0.0}, {"alpha": -1e-3}, {"alpha": 1e-12}, {"alpha": 1e40}, {"scale": 1e299}, {"scale": numpy.inf},
           {"position": 1e9}, {"position": numpy.nan}, {"coeff": numpy.inf}, {"coeff": numpy.nan}, {"coeff": 1.7e308},
           {"row": 1e-290}]


@pytest.mark.parametrize("what", ["rho", "grad", "laplacian", "mo"])
@pytest.mark.parametrize("change", OUTSIDE, ids=str)
def test_parameters_beyond_the_digits(core, what, change):
    qc = edit(molecule("d"), **change)
    pts = near_points(qc, 5003)
    pts[:, ~numpy.isfinite(pts).all(axis=0)] = 0.5
    compare(core, qc, what, pts)


def device_call(core, qc, pts):
    import torch
    from orbkit_gb300 import _lib
    dev = torch.device("cuda")
    b = core.get_basis(qc.geo_spec, qc.ao_spec, dev)
    C = b.c_eff(qc.mo_spec.get_coeffs())
    occ = torch.as_tensor(qc.mo_spec.get_occ(), dtype=torch.float64, device=dev).contiguous()
    xyz = torch.as_tensor(pts, device=dev).contiguous()
    n = pts.shape[1]
    return b, C, occ, xyz, _lib.OkgGrid(xyz[0].data_ptr(), xyz[1].data_ptr(), xyz[2].data_ptr(), n, 0, 0, 0, 0, 0), n


@pytest.mark.parametrize("change", [{}, {"scale": 1e299, "coeff": 0.0}], ids=str)
def test_norms_are_added_once(core, change):
    """The MO norms of a call, also of one whose tiles find AO values beyond the digits."""
    import torch
    from orbkit_gb300 import _lib
    L = _lib.load()
    qc = edit(molecule("p"), **change)
    pts = near_points(qc, 6000)
    b, C, occ, xyz, gd, n = device_call(core, qc, pts)
    C[:, 2:] *= 1e-160 if change else 1.0
    mo = torch.empty((7, n), dtype=torch.float64, device=C.device)
    _lib.check(L.okg_eval_mo(b.handle, gd, 7, _lib.ptr(C), 1, _lib.int_array([0]), 0, _lib.ptr(mo), n, _lib.stream_handle()))
    norm = torch.ones(7, dtype=torch.float64, device=C.device)
    rho = torch.empty(n, dtype=torch.float64, device=C.device)
    _lib.check(L.okg_rho(b.handle, gd, 7, _lib.ptr(C), _lib.ptr(occ), 0, _lib.int_array([]), 0, _lib.ptr(rho), None, n,
                         _lib.ptr(norm), _lib.stream_handle()))
    want = 1.0 + (mo ** 2).sum(1)
    assert torch.isfinite(want).all()
    assert (torch.abs(norm - want) <= 1e-12 * want).all()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("change", [{}, {"alpha": -1e-3}, {"coeff": numpy.inf}, {"coeff": numpy.nan}, {"cotangent": numpy.inf},
                                    {"cotangent": numpy.nan}, {"gradient": -numpy.inf}], ids=str)
def test_adjoint_beyond_the_digits(core, precision, change):
    """The whole workspace (pipeline) against one that only fits the one-kernel form: its bits
    where the pipeline leaves the call to that form."""
    import ctypes
    import torch
    from orbkit_gb300 import _lib, adjoint
    L = adjoint._L()
    cot = {k: v for k, v in change.items() if k in ("cotangent", "gradient")}
    qc = edit(molecule("d"), **{k: v for k, v in change.items() if k not in cot})
    pts = near_points(qc, 4100)
    b, C, occ, xyz, gd, n = device_call(core, qc, pts)
    gen = torch.Generator(device=C.device).manual_seed(3)
    g = torch.randn((4, n), generator=gen, dtype=torch.float64, device=C.device)
    if "cotangent" in cot:
        g[0, 700] = cot["cotangent"]
    if "gradient" in cot:
        g[2, 4000] = cot["gradient"]
    size = ctypes.c_size_t(0)
    _lib.check(L.okg_rho_backward_workspace(b.handle, gd, 7, precision, ctypes.byref(size)))

    def run(nbytes):
        work = torch.full((nbytes,), 255, dtype=torch.uint8, device=C.device)
        out = [torch.empty(s, dtype=torch.float64, device=C.device) for s in (tuple(C.shape), (b.nprim, 2), (b.natom, 3))]
        _lib.check(L.okg_rho_backward(b.handle, gd, 7, _lib.ptr(C), _lib.ptr(occ), _lib.ptr(g[0]), _lib.ptr(g[1]), n, precision,
                                      *[_lib.ptr(o) for o in out], _lib.ptr(work), nbytes, _lib.stream_handle()))
        return out

    for u, v in zip(run(size.value), run(size.value - 256)):
        if change:
            assert not torch.isfinite(v).all() or "alpha" in change
            assert torch.equal(torch.nan_to_num(u, 7.0, 8.0, 9.0), torch.nan_to_num(v, 7.0, 8.0, 9.0))
            assert torch.equal(torch.isnan(u), torch.isnan(v))
        else:
            assert torch.isfinite(u).all()
