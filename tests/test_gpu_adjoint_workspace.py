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
