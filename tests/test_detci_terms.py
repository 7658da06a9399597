"""detCI term lists: what the conversion in one go takes is what the entry-by-entry one gives, and
what that refuses is refused."""
import numpy
import pytest

torch = pytest.importorskip("torch")
from orbkit_gb300 import detci  # noqa: E402


def entry_by_entry(sing):
    coef = numpy.asarray([float(c) for c in sing[0]], dtype=numpy.float64)
    pairs = numpy.asarray([[int(p[0]), int(p[1])] for p in sing[1]], dtype=numpy.int32).reshape(-1, 2)
    return coef, pairs


class OnDevice:
    """Numbers that numpy cannot read as an array (a tensor on a device)."""

    def __init__(self, values):
        self.values = values

    def __array__(self, *a, **k):
        raise TypeError("can't convert cuda:0 device type tensor to numpy")

    def __len__(self):
        return len(self.values)

    def __getitem__(self, i):
        return self.values[i]


I32 = 2 ** 31
FORMS = [
    [[0.5, -2], [[0, 1], [2, 3]]], [[1, 2], [(0, 1), (2, 3)]], [[], []], [[0.5], [[I32 - 1, -I32]]],
    [numpy.float32([0.1, 0.2]), numpy.int64([[0, 1], [5, 4]])], [numpy.uint8([3]), numpy.uint64([[1, 2]])],
    [[True, 2.0], [[True, 0], [1, 1]]], [[0.5], [[1.9, 2.1]]], [[0.5], [[1, 2, 3]]], [["0.5"], [["1", "2"]]],
    [[0.5, 0.25], [[1, 2], [3, 4, 5]]], [[0.5], [numpy.array([[1], [2]])]], [[0.5, 1.0], [[1, 2]]],
    [torch.tensor([0.5, 1.0], requires_grad=True), torch.tensor([[0, 1], [1, 0]])], [OnDevice([0.5, 1.0]), OnDevice([[0, 1], [2, 3]])],
    [numpy.float64([0.5, 1.0])[::-1], numpy.int32([[1, 2], [3, 4]]).T], [[10 ** 400], [[0, 1]]], [[1j], [[0, 1]]], [[None], [[0, 1]]],
    [[0.5], [[I32, 0]]], [[0.5], [[0, 2 ** 32 + 1]]], [[0.5], numpy.int64([[0, -I32 - 1]])], [[0.5], numpy.uint64([[2 ** 63, 0]])],
    [[0.5], [[2 ** 70, 0]]], [[0.5], [[1]]], [[0.5], [1, 2]],
]


@pytest.mark.parametrize("k", range(len(FORMS)))
def test_same_as_entry_by_entry(k):
    def outcome(f):
        try:
            return f(FORMS[k])
        except Exception as e:
            return type(e)

    a, b = outcome(detci._sing_terms), outcome(entry_by_entry)
    if isinstance(b, type):
        assert a is b
        return
    for u, v in zip(a, b):
        assert u.dtype == v.dtype and u.shape == v.shape and (u == v).all()
