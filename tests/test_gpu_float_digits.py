"""Single-precision digits of the FP32 adjoint: values far below the largest of their 64 points
count as nothing, not as a whole unit of the last digit."""
import ctypes

import numpy
import pytest

from test_gpu_split64_range import device_call

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


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("small", [1e-10, 1e-12, 1e-30])
def test_small_values_of_a_block(core, small, sign):
    """One s function; in every block of 64 points one with the function at its largest and
    cotangent 0, the others with the function at `small` of it.  dL/dC is the sum of
    (2 occ g MO) chi over the others.  A chi is off by half a unit, 2^-32 of the largest, at
    most, and where it is below a quarter of a unit by itself alone."""
    import torch
    from orbkit_gb300 import _lib, adjoint, synthetic
    from orbkit_gb300.orbitals import AOClass, MOClass
    L = adjoint._L()
    ao = AOClass([{"atom": 0, "type": "s", "pnum": 1, "coeffs": numpy.array([[1.0, 1.0]])}])
    ao.update()
    mo = MOClass([{"coeffs": numpy.array([sign]), "occ_num": 1.0, "energy": 0.0, "sym": "1.1"}])
    mo.update()
    qc = synthetic.make_qc(numpy.zeros((1, 3)), ["C"], ao, mo)
    pts = numpy.zeros((3, 4096))
    pts[0] = numpy.sqrt(-numpy.log(small))
    pts[0, ::64] = 0.0
    b, C, occ, xyz, gd, n = device_call(core, qc, pts)
    g = torch.ones(n, dtype=torch.float64, device="cuda")
    g[::64] = 0.0

    def run(precision):
        size = ctypes.c_size_t(0)
        _lib.check(L.okg_rho_backward_workspace(b.handle, gd, 1, precision, ctypes.byref(size)))
        work = torch.empty(size.value, dtype=torch.uint8, device="cuda")
        out = [torch.empty(s, dtype=torch.float64, device="cuda") for s in ((1, 1), (1, 2), (1, 3))]
        _lib.check(L.okg_rho_backward(b.handle, gd, 1, _lib.ptr(C), _lib.ptr(occ), _lib.ptr(g), None, n, precision,
                                      *[_lib.ptr(o) for o in out], _lib.ptr(work), size.value, _lib.stream_handle()))
        return float(out[0])

    chi = core.ao_creator(qc.geo_spec, qc.ao_spec, x=pts[0], y=pts[1], z=pts[2], is_vector=True)[0]
    exact = sign * 2.0 * (g.cpu().numpy() * chi * chi).sum()
    unit = 2.0 ** -31 * chi.max()
    off = numpy.where(chi < unit / 4, chi, unit / 2)
    assert abs(run(32) - exact) <= 1.01 * (2.0 * g.cpu().numpy() * chi * off).sum()
