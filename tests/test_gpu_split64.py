"""The tensor-core FP64 path (okg_split64.cu): large okg_rho / okg_eval_mo calls against
the oracle, and against the DFMA kernel (the same points in small calls).

Bar: the FP64 parity bar of every FP64 output (helpers.FP64_*).
"""
import ctypes

import numpy
import pytest

from helpers import FP64_ATOL_REL, FP64_RTOL, assert_fp64_close

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


def molecule(nmo, seed=0, natom=5, top="g", spherical=False):
    """Random molecule with every shell type up to `top`, steep and diffuse primitives and
    contractions of 1 to 7 primitives of either sign."""
    from orbkit_gb300 import synthetic
    from orbkit_gb300.orbitals import AOClass, MOClass
    rng = numpy.random.default_rng(seed)
    geo = synthetic.random_geometry(rng, natom, 6.0)
    ao = []
    for a in range(natom):
        for lt in "spdfg"[:"spdfg".index(top) + 1]:
            for n in ((7, 1) if lt == "s" else (2,)):
                alpha = numpy.exp(rng.uniform(numpy.log(0.05), numpy.log(5e4 if lt == "s" else 30.0), n))
                ao.append({"atom": a, "type": lt, "pnum": n,
                           "coeffs": numpy.stack([alpha, rng.uniform(-1.0, 1.0, n)], axis=1)})
    spec = AOClass(ao)
    if spherical:
        spec.set_lm_dict(p=[1, 0])
    spec.update()
    C = rng.standard_normal((nmo, spec.get_ao_num())) * numpy.exp(rng.uniform(-6, 2, (nmo, 1)))
    occ = numpy.where(rng.random(nmo) < 0.5, 2.0, rng.uniform(-1.0, 2.0, nmo))
    mo = MOClass([{"coeffs": C[i], "occ_num": float(occ[i]), "energy": 0.0, "sym": "%d.1" % (i + 1)} for i in range(nmo)])
    mo.update()
    return synthetic.make_qc(geo, ["C"] * natom, spec, mo)


def call(core, qc, what, *grid, vec=True):
    if what == "mo":
        return [core.rho_compute_no_slice(qc, calc_mo=True, x=grid[0], y=grid[1], z=grid[2], is_vector=vec)]
    more = {"rho": {}, "grad": {"drv": ["x", "y", "z"]}, "laplacian": {"laplacian": True},
            "mixed_orders": {"drv": ["zz", "x", "yy", "x"]}}[what]
    out = core.rho_compute_no_slice(qc, x=grid[0], y=grid[1], z=grid[2], is_vector=vec, **more)
    return list(out) if isinstance(out, tuple) else [out]


def reference(qc, what, *grid, vec=True):
    okref = pytest.importorskip("okref")
    more = {"rho": {}, "grad": {"drv": ["x", "y", "z"]}, "laplacian": {"laplacian": True},
            "mixed_orders": {"drv": ["zz", "x", "yy", "x"]}, "mo": {"calc_mo": True}}[what]
    out = okref.rho_compute_no_slice(qc, x=grid[0], y=grid[1], z=grid[2], is_vector=vec, **more)
    return list(out) if isinstance(out, tuple) else [out]


@pytest.mark.parametrize("what", ["rho", "grad", "laplacian", "mixed_orders", "mo"])
@pytest.mark.parametrize("nmo,npts,spherical", [(1, 4864, False), (16, 4865, True), (17, 4991, False), (33, 5003, True),
                                                (65, 4896, False), (130, 4897, False)])
def test_vector_points_vs_oracle(core, what, nmo, npts, spherical):
    """Operand-column edges (16, 64, several passes), ragged point counts."""
    qc = molecule(nmo, seed=nmo, top="f" if spherical else "g", spherical=spherical)
    pts = numpy.random.default_rng(npts).uniform(-6.0, 6.0, (3, npts))
    pts[:, :5] = numpy.asarray(qc.geo_spec).T  # the nuclei themselves
    for a, b in zip(call(core, qc, what, *pts), reference(qc, what, *pts)):
        assert_fp64_close(a, b, "%s nmo=%d" % (what, nmo))


@pytest.mark.parametrize("shape", [(1, 1, 4999), (23, 9, 31), (4, 160, 8), (70, 5, 15)])
def test_regular_grids_vs_oracle(core, shape):
    """Bricks at the grid's edges, 32- and 128-point tiles."""
    qc = molecule(9, seed=3)
    axes = [numpy.linspace(-4.0, 5.0, n) for n in shape]
    for what in ("rho", "grad", "laplacian", "mo"):
        for a, b in zip(call(core, qc, what, *axes, vec=False), reference(qc, what, *axes, vec=False)):
            assert_fp64_close(a, b, "%s %s" % (what, shape))


def both_routes(core, qc, what, pts):
    """The call whole (tensor cores) and in runs of 300 points (DFMA kernel)."""
    whole = call(core, qc, what, *pts)
    runs = [call(core, qc, what, *pts[:, i:i + 300]) for i in range(0, pts.shape[1], 300)]
    return whole, [numpy.concatenate([r[k] for r in runs], axis=-1) for k in range(len(whole))]


@pytest.mark.parametrize("what", ["rho", "grad", "laplacian", "mo"])
def test_far_and_non_finite_points(core, what):
    """Points far from every atom (values down to zero), huge and non-finite coordinates:
    the same as the DFMA kernel, and the points that share their tiles are not affected."""
    qc = molecule(6, seed=11, top="p")
    rng = numpy.random.default_rng(4)
    pts = rng.uniform(-5.0, 5.0, (3, 6000))
    pts[:, ::7] *= 10.0 ** rng.uniform(0.0, 3.5, len(pts[0, ::7]))
    pts[0, 100], pts[1, 333], pts[2, 2000], pts[0, 4001] = 1e19, -1e25, numpy.nan, numpy.inf
    a, b = both_routes(core, qc, what, pts)
    for u, v in zip(a, b):
        assert numpy.array_equal(numpy.isnan(u), numpy.isnan(v))
        m = ~numpy.isnan(v)
        assert (numpy.abs(u[m] - v[m]) <= FP64_RTOL * numpy.abs(v[m]) + FP64_ATOL_REL * numpy.abs(v[m]).max()).all()


def test_non_finite_parameters(core):
    """NaN and zero MO coefficients and a NaN position: NaN where the DFMA kernel has it."""
    pts = numpy.random.default_rng(5).uniform(-5.0, 5.0, (3, 5000))
    qc = molecule(20, seed=12, top="d")
    qc.mo_spec[3]["coeffs"] = qc.mo_spec[3]["coeffs"] * numpy.nan
    qc.mo_spec[7]["coeffs"] = qc.mo_spec[7]["coeffs"] * 0.0
    qc.mo_spec.update()
    a, b = both_routes(core, qc, "mo", pts)
    assert numpy.isnan(a[0][3]).all() and (a[0][7] == 0).all()
    keep = [i for i in range(20) if i != 3]
    assert_fp64_close(a[0][keep], b[0][keep], "other MOs")
    a, b = both_routes(core, qc, "grad", pts)
    assert all(numpy.isnan(u).all() and numpy.isnan(v).all() for u, v in zip(a, b))
    qc = molecule(20, seed=12, top="d")
    qc.geo_spec[1, 2] = numpy.nan
    a, b = both_routes(core, qc, "rho", pts)
    assert numpy.isnan(a[0]).all() and numpy.isnan(b[0]).all()


def test_norms_streams_and_capture(core):
    """MO norms against the MO grid; two streams at once; a captured call (the DFMA kernel)
    agrees with the plain one; no wait expired."""
    import torch
    from orbkit_gb300 import _lib
    L = _lib.load()
    qc = molecule(50, seed=13, top="d")
    dev = torch.device("cuda")
    b = core.get_basis(qc.geo_spec, qc.ao_spec, dev)
    C = b.c_eff(qc.mo_spec.get_coeffs())
    occ = torch.as_tensor(qc.mo_spec.get_occ(), dtype=torch.float64, device=dev).contiguous()
    n = 6001
    pts = torch.rand((3, n), dtype=torch.float64, device=dev) * 8.0 - 4.0
    gd = _lib.OkgGrid(pts[0].data_ptr(), pts[1].data_ptr(), pts[2].data_ptr(), n, 0, 0, 0, 0, 0)

    def run(stream, norm=None):
        rho = torch.empty(n, dtype=torch.float64, device=dev)
        grad = torch.empty((3, n), dtype=torch.float64, device=dev)
        codes = _lib.int_array([1, 2, 3])
        _lib.check(L.okg_rho(b.handle, gd, 50, _lib.ptr(C), _lib.ptr(occ), 3, codes, 0, _lib.ptr(rho), _lib.ptr(grad), n,
                             _lib.ptr(norm), _lib.stream_handle(stream)))
        return rho, grad

    cur = torch.cuda.current_stream()
    norm = torch.zeros(50, dtype=torch.float64, device=dev)
    r0, g0 = run(cur, norm)
    x, y, z = pts.cpu().numpy()
    mo = core.rho_compute_no_slice(qc, calc_mo=True, x=x, y=y, z=z, is_vector=True)
    assert_fp64_close(norm.cpu().numpy(), (mo ** 2).sum(1), "norms")
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [run(s) for s in streams for _ in range(3)]
    torch.cuda.synchronize()
    for r, g in outs:
        assert torch.equal(r, r0) and torch.equal(g, g0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r1, g1 = run(torch.cuda.current_stream())
    graph.replay()
    torch.cuda.synchronize()
    assert_fp64_close(r1.cpu().numpy(), r0.cpu().numpy(), "captured rho")
    assert_fp64_close(g1.cpu().numpy(), g0.cpu().numpy(), "captured gradient")
    st = ctypes.c_int(7)
    assert L.okg_wait_status(ctypes.byref(st)) == 0 and st.value == 0
