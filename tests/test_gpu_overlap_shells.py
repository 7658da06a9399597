"""The overlap kernels' routes give the same bits: ket shells in the canonical component
order (shell kernel) against explicit lists in another order (element kernel), one geometry
tensor (symmetric pair table) against two equal ones."""
import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 1, 1, 1, 1), (7, 2, 3, 1, 2), (33, 0, 0, 0, 0), (1, 32, 0, 33, 0)])
def test_routes_agree(counts):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orbkit_gb300 import build
    build.build()
    from orbkit_gb300.analytical_integrals import OverlapPlan
    from orbkit_gb300.orbitals import AOClass
    from orbkit_gb300.tools import cartesian_order
    rng = numpy.random.default_rng(sum(counts))
    shells, perm, row = [], [], 0
    for l, n in enumerate(counts):
        for _ in range(n):
            k = int(rng.integers(1, 5))
            alpha = numpy.exp(rng.uniform(-3.0, 7.0, k))
            shells.append({"atom": int(rng.integers(3)), "type": "spdfg"[l], "pnum": k,
                           "coeffs": numpy.stack([alpha, rng.uniform(-1.0, 1.0, k)], axis=1)})
            nc = len(cartesian_order[l])
            perm.extend(row + numpy.arange(nc)[::-1])
            row += nc
    shells[0]["atom"] = 2  # (every atom below the largest used exists)
    listed = [dict(s, lxlylz=cartesian_order["spdfg".index(s["type"])][::-1]) for s in shells]
    plans = []
    for data in (shells, listed):
        spec = AOClass(data)
        spec.update()
        plans.append(OverlapPlan(spec))
    geo = torch.as_tensor(rng.uniform(-3.0, 3.0, (3, 3)), device="cuda")
    idx = torch.as_tensor(numpy.array(perm), device="cuda")
    for drv in range(4):
        a = plans[0].run(geo, geo, drv)
        assert torch.equal(a, plans[0].run(geo, geo.clone(), drv)), "pair table, drv %d" % drv
        b = plans[1].run(geo, geo, drv)
        assert torch.equal(a[idx][:, idx], b), "shell and element kernels, drv %d" % drv
