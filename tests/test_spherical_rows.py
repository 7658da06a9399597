"""Spherical rows of shells that the basis does not have are refused."""
import numpy
import pytest

from orbkit_gb300.basis import spherical_csr


class Listing:
    """Two p shells and a spherical row of `shell`."""

    def __init__(self, shell):
        self.shell = shell

    def get_lxlylz(self):
        return numpy.array([[1, 0, 0], [0, 1, 0], [0, 0, 1]] * 2)

    def get_assign_lxlylz_to_cont(self):
        return [0] * 3 + [1] * 3

    def get_old_ao_spherical(self):
        return [[0, (1, 0)], [self.shell, (1, 1)]]


@pytest.mark.parametrize("shell", [-3, -2, -1, 2, 7])
def test_unknown_shell(shell):
    with pytest.raises(KeyError):
        spherical_csr(Listing(shell))


def test_known_shells():
    for shell in (0, 1):
        ptr, idx, coef = spherical_csr(Listing(shell))
        assert list(ptr) == [0, 1, 2] and list(idx) == [2, 3 * shell] and (coef == 1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("spherical", [False, True])
def test_dense_transform_on_host_and_device(spherical):
    torch = pytest.importorskip("torch")
    from orbkit_gb300 import synthetic
    from orbkit_gb300.basis import DeviceBasis
    rng = numpy.random.default_rng(1)
    spec = synthetic.build_basis(rng, ["C", "H"], with_f=True, spherical=spherical)
    b = DeviceBasis(rng.uniform(-1.0, 1.0, (2, 3)), spec, torch.device("cuda"))
    if not spherical:
        assert b.T is None and b.T_dev is None
        return
    assert b.T.shape == (b.nao, b.ncart) and numpy.array_equal(b.T_dev.cpu().numpy(), b.T) and b.T_dev.is_cuda
    C = rng.standard_normal((3, b.nao))
    assert numpy.abs(b.c_eff(C).cpu().numpy() - C @ b.T).max() <= 1e-14 * numpy.abs(C).sum(1).max()
