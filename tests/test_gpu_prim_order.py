"""The per-shell ordering of primitives on the device (okg_basis_set_params): shells of 1 to
40 primitives, equal exponents, and exponents in any order give the same density as the same
primitives given in ascending order.

Bar: the FP64 parity bar (only the order of the radial sums differs), and the oracle.
"""
import numpy
import pytest

from helpers import assert_fp64_close
from test_gpu_split64 import call, core, reference  # noqa: F401  (core: the fixture)

pytestmark = pytest.mark.gpu


def molecule(order):
    from orbkit_gb300 import synthetic
    from orbkit_gb300.orbitals import AOClass, MOClass
    rng = numpy.random.default_rng(2)
    geo = synthetic.random_geometry(rng, 6, 6.0)
    ao = []
    for atom, n in enumerate((1, 2, 31, 32, 33, 40)):
        for lt in "sp":
            alpha = numpy.round(numpy.exp(rng.uniform(-2.0, 5.0, n)), 1) + 0.1  # some are equal
            prim = numpy.stack([alpha, rng.uniform(-1.0, 1.0, n)], axis=1)
            if order == "ascending":
                prim = prim[numpy.argsort(alpha, kind="stable")]
            ao.append({"atom": atom, "type": lt, "pnum": n, "coeffs": prim})
    spec = AOClass(ao)
    spec.update()
    C = rng.standard_normal((5, spec.get_ao_num()))
    mo = MOClass([{"coeffs": C[i], "occ_num": 2.0, "energy": 0.0, "sym": "%d.1" % (i + 1)} for i in range(5)])
    mo.update()
    return synthetic.make_qc(geo, ["C"] * 6, spec, mo)


@pytest.mark.parametrize("what", ["rho", "grad"])
def test_order_of_primitives(core, what):  # noqa: F811
    pts = numpy.random.default_rng(3).uniform(-5.0, 5.0, (3, 6000))
    given, ascending = molecule("given"), molecule("ascending")
    a, b = call(core, given, what, *pts), call(core, ascending, what, *pts)
    for u, v, r in zip(a, b, reference(given, what, *pts)):
        assert_fp64_close(u, v, what)
        assert_fp64_close(u, r, what)
