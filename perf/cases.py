"""Performance cases: the grid evaluations, fits and integrals that a program built on
this package has it do, each through the entry points such a program calls.

Molecules are seeded and synthetic (orbkit_gb300.synthetic's shell recipe, exponent
ranges and box sizes); the seed changes the geometry, the exponents and the
coefficients, the case fixes the sizes.  ``exact`` restates the definitions in plain
torch and numpy in 64 bits.
"""
import math

import numpy
import torch

from orbkit_gb300 import analytical_integrals, core, detci, synthetic
from orbkit_gb300 import grid as okgrid
from orbkit_gb300.adjoint import DensityModel, density_fit_loss
from orbkit_gb300.batch import BatchEvaluator


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # Density at a handful of points (a bond midpoint, a critical-point search): one
        # small call after another, so launches and host work are what counts.
        {"name": "density_few_points", "kind": "density", "what": "rho", "atoms": 3, "basis": "cart", "grid": "points",
         "npts": 27, "precision": "fp64"},
        # The first thing a user runs: the density of a small molecule on a cube grid, with
        # the defaults (the package's small configuration: 3 atoms, 25 AOs, 5 MOs, 80^3).
        {"name": "density_water_cube", "kind": "density", "what": "rho", "atoms": 3, "basis": "cart", "grid": "regular",
         "nx": 80, "ny": 80, "nz": 80, "precision": "fp64"},
        # Density and gradient in double precision on a fine grid of a mid-size molecule
        # (the benchmark's 20-atom, 180-AO, 40-MO molecule on 160^3 points).
        {"name": "density_gradient_fp64", "kind": "density", "what": "grad", "atoms": 20, "basis": "cart",
         "grid": "regular", "nx": 160, "ny": 160, "nz": 160, "precision": "fp64"},
        # Density and Laplacian for a topology analysis: a spherical basis with f shells on
        # a box with three different, ragged edges.
        {"name": "laplacian_spherical", "kind": "density", "what": "laplacian", "atoms": 12, "basis": "sph",
         "grid": "regular", "nx": 61, "ny": 83, "nz": 47, "precision": "fp64"},
        # Density and gradient of a large molecule (200 atoms, f shells, spherical, 400 MOs)
        # on an odd number of atom-centred quadrature points.
        {"name": "density_large_points", "kind": "density", "what": "grad", "atoms": 200, "basis": "sph",
         "grid": "points", "npts": 20011, "precision": "fp64"},
        # The same mid-size molecule and grid on the mixed-precision path (the benchmark's
        # headline workload), results on the host as the drop-in returns them.
        {"name": "density_gradient_mixed", "kind": "density", "what": "grad", "atoms": 20, "basis": "cart",
         "grid": "regular", "nx": 160, "ny": 160, "nz": 160, "precision": "mixed"},
        # Orbital cubes for plotting: every occupied MO on a grid.
        {"name": "mo_cubes", "kind": "mo", "atoms": 20, "basis": "cart", "grid": "regular", "nx": 80, "ny": 80,
         "nz": 80},
        # One optimisation step of a density fit in double precision: loss and gradients
        # with respect to coefficients, exponents and positions.
        {"name": "fit_step_fp64", "kind": "fit", "atoms": 12, "nx": 64, "ny": 64, "nz": 64, "precision": "fp64"},
        # The same in single precision (float32 parameters) on the finer grid that is
        # usual there.
        {"name": "fit_step_fp32", "kind": "fit", "atoms": 12, "nx": 104, "ny": 96, "nz": 101, "precision": "fp32"},
        # Many molecules with atom-centred point sets in one launch (dataset generation).
        {"name": "batch_molecules", "kind": "batch", "molecules": 16, "min_atoms": 3, "max_atoms": 30, "radial": 60,
         "angular": 151},
        # AO overlap and its three ket derivatives with a plan kept across geometries
        # (a geometry scan): 120 atoms, f shells, spherical.
        {"name": "overlap_derivatives", "kind": "overlap", "atoms": 120, "basis": "sph"},
        # detCI transition density and flux density from MO grids that are already on the
        # device.
        {"name": "detci_density_flux", "kind": "detci", "nmo": 42, "npts": 1048576, "zero": 436, "sing": 7160},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _edges(rng, npts):
    """Three edges, usually different and odd, with about npts points in all."""
    a = npts ** (1.0 / 3.0)
    nx = max(2, int(round(a * rng.uniform(0.7, 1.4))))
    ny = max(2, int(round(a * rng.uniform(0.7, 1.4))))
    nz = max(2, int(npts / float(nx * ny)))
    return {"nx": nx, "ny": ny, "nz": nz}


def draw(rng):
    kind = rng.choice(["density", "density", "density", "mixed", "mo", "ao", "fit", "fit", "batch", "overlap", "detci"])
    basis = rng.choice(["cart", "sph"])
    if kind in ("density", "mixed"):
        atoms = _log(rng, 3, 200)
        what = "grad" if kind == "mixed" else rng.choice(["rho", "grad", "laplacian"])
        # double precision: no more arithmetic than the largest listed case
        most = 3.0e6 if kind == "mixed" else min(3.0e6, 6.0e10 / (2.0 * _nao(atoms, basis) * _nmo(atoms) * 7))
        most /= max(1.0, (atoms / 30.0) ** 2) if kind == "mixed" else 1.0
        if kind == "mixed":
            low = min(20000, int(most))
        else:
            low = min(200, int(most))
        npts = _log(rng, low, int(most))
        c = {"kind": "density", "what": what, "atoms": atoms, "basis": basis,
             "precision": "mixed" if kind == "mixed" else "fp64"}
        if kind == "density" and rng.random() < 0.4:
            npts = min(npts, 400000)
            c.update({"grid": "points", "npts": npts})
        else:
            c.update({"grid": "regular"}, **_edges(rng, npts))
        return c
    if kind in ("mo", "ao"):
        atoms = _log(rng, 3, 40)
        rows = _nmo(atoms) if kind == "mo" else _nao(atoms, basis)
        npts = _log(rng, 1000, int(1.5e7 / rows))
        return dict({"kind": kind, "atoms": atoms, "basis": basis, "grid": "regular"}, **_edges(rng, npts))
    if kind == "fit":
        prec = rng.choice(["fp64", "fp32"])
        atoms = _log(rng, 3, 20)
        most = (2.0e5 if prec == "fp64" else 8.0e5) * min(1.0, (12.0 / atoms) ** 2)
        return dict({"kind": "fit", "atoms": atoms, "precision": prec}, **_edges(rng, _log(rng, 4000, int(most))))
    if kind == "batch":
        hi = _log(rng, 6, 30)
        return {"kind": "batch", "molecules": _log(rng, 2, 16), "min_atoms": 3, "max_atoms": hi,
                "radial": rng.randint(40, 60), "angular": rng.randint(90, 151)}
    if kind == "overlap":
        return {"kind": "overlap", "atoms": _log(rng, 3, 110), "basis": basis}
    zero = _log(rng, 20, 436)
    return {"kind": "detci", "nmo": rng.randint(8, 42), "npts": _log(rng, 1000, 1000000), "zero": zero,
            "sing": _log(rng, 20, 7000)}


# ------------------------------------------------------------------ molecules
def _elements(atoms):
    """Two heavy atoms in five (the recipe's 8 in 20), the first one heavy."""
    return ["O" if i % 5 == 0 else "C" if i % 5 == 2 else "H" for i in range(atoms)]


def _heavy(atoms):
    return sum(e != "H" for e in _elements(atoms))


def _nao(atoms, basis):
    heavy = _heavy(atoms)
    return heavy * (15 if basis == "cart" else 21) + 5 * (atoms - heavy)


def _nmo(atoms):
    return 5 if atoms == 3 else 2 * atoms


def _ncart(atoms, basis):
    heavy = _heavy(atoms)
    return heavy * (15 if basis == "cart" else 25) + 5 * (atoms - heavy)


def _molecule(atoms, basis, seed):
    rng = numpy.random.default_rng(seed)
    if atoms == 3:  # water-like, as the package's small configuration
        half = numpy.deg2rad(104.5) / 2.0
        geo = numpy.array([[0.0, 0.0, 0.0], [0.0, 1.81 * numpy.sin(half), 1.81 * numpy.cos(half)],
                           [0.0, -1.81 * numpy.sin(half), 1.81 * numpy.cos(half)]])
        geo = geo + 0.05 * rng.standard_normal(geo.shape)
    else:
        geo = synthetic.random_geometry(rng, atoms, _box(atoms))
    el = _elements(atoms)
    ao = synthetic.build_basis(rng, el, with_f=basis == "sph", spherical=basis == "sph")
    # overlap-orthonormal MOs; above 60 atoms orthonormal coefficient rows (the host
    # overlap of a large basis takes seconds)
    S = None if atoms <= 60 else numpy.eye(ao.get_ao_num())
    mo = synthetic.build_mos(rng, geo, ao, _nmo(atoms), S=S)
    return rng, synthetic.make_qc(geo, el, ao, mo)


def _box(atoms):
    return 16.0 * (atoms / 20.0) ** (1.0 / 3.0)


def _axes(case):
    half = _box(case["atoms"]) / 2.0 + (2.5 if case["atoms"] == 3 else 4.0)
    return [numpy.linspace(-half, half, case[k]) for k in ("nx", "ny", "nz")]


def _points(case, rng, geo):
    """Atom-centred quadrature points, exactly case['npts'] of them in all."""
    n = case["npts"]
    per = -(-n // len(geo))
    nr = min(50, max(3, per // 8))
    r = synthetic.becke_radial(nr)
    u = synthetic.fibonacci_sphere(-(-per // nr))
    shell = (r[:, None, None] * u[None, :, :]).reshape(-1, 3)
    pts = (geo[:, None, :] + shell[None, :, :]).reshape(-1, 3)
    return numpy.ascontiguousarray(pts[numpy.sort(rng.permutation(len(pts))[:n])].T)


def _npts(case):
    return case["npts"] if case.get("grid") == "points" else case["nx"] * case["ny"] * case["nz"]


# ------------------------------------------------------------------ the interface
def prepare(case, seed):
    core.quiet = True  # a program that wants no terminal output
    kind = case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    if kind in ("density", "mo", "ao"):
        rng, qc = _molecule(case["atoms"], case["basis"], seed)
        st = {"case": case, "qc": qc}
        if case["grid"] == "points":
            st["points"] = _points(case, rng, qc.geo_spec)
        else:
            st["axes"] = _axes(case)
        return st
    if kind == "fit":
        rng, qc = _molecule(case["atoms"], "cart", seed)
        axes = _axes(case)
        dt = torch.float64 if case["precision"] == "fp64" else torch.float32
        leaf = lambda a: torch.tensor(numpy.asarray(a), dtype=dt, device=dev, requires_grad=True)
        prim = qc.ao_spec.get_prim_coeffs()
        st = {"case": case, "qc": qc, "axes": axes, "model": DensityModel(qc, *axes, False, case["precision"])}
        st["params"] = [leaf(qc.mo_spec.get_coeffs()), leaf(prim[:, 0]), leaf(prim[:, 1]), leaf(qc.geo_spec)]
        st["target"] = _promolecule(qc.geo_spec, axes, dev)
        gen = torch.Generator(device=dev).manual_seed(seed)
        st["weights"] = torch.rand(_npts(case), generator=gen, dtype=torch.float64, device=dev)
        return st
    if kind == "batch":
        mols = []
        for i in range(case["molecules"]):
            span = case["max_atoms"] - case["min_atoms"]
            atoms = case["min_atoms"] + (i * span) // max(1, case["molecules"] - 1)
            rng, qc = _molecule(atoms, "cart", [seed, i])
            shell = (synthetic.becke_radial(case["radial"])[:, None, None] *
                     synthetic.fibonacci_sphere(case["angular"])[None]).reshape(-1, 3)
            mols.append((qc, numpy.ascontiguousarray((qc.geo_spec[:, None] + shell[None]).reshape(-1, 3).T)))
        return {"case": case, "mols": mols, "batch": BatchEvaluator(mols, tune=False)}
    if kind == "overlap":
        _, qc = _molecule(case["atoms"], case["basis"], seed)
        return {"case": case, "qc": qc, "plan": analytical_integrals.OverlapPlan(qc.ao_spec),
                "geo": torch.tensor(qc.geo_spec, dtype=torch.float64, device=dev)}
    if kind == "detci":
        gen = torch.Generator(device=dev).manual_seed(seed)
        nmo, npts = case["nmo"], case["npts"]
        rng = numpy.random.default_rng(seed)
        z = [[list(rng.standard_normal(1)) for _ in range(case["zero"])],
             [[int(rng.integers(nmo))] for _ in range(case["zero"])]]
        pairs = rng.integers(0, nmo, (case["sing"], 2))
        s = [list(rng.standard_normal(case["sing"])), [[int(a), int(b)] for a, b in pairs]]
        return {"case": case, "zero": z, "sing": s,
                "mo": torch.randn((nmo, npts), generator=gen, dtype=torch.float64, device=dev),
                "drv": torch.randn((3, nmo, npts), generator=gen, dtype=torch.float64, device=dev)}
    raise ValueError(kind)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "density":
        drv = ["x", "y", "z"] if case["what"] == "grad" else None
        more = {"drv": drv, "laplacian": case["what"] == "laplacian", "precision": case["precision"]}
        if case["grid"] == "points":
            x, y, z = st["points"]
            return core.rho_compute_no_slice(st["qc"], x=x, y=y, z=z, is_vector=True, **more)
        okgrid.set_grid(*st["axes"], is_vector=False)
        return core.rho_compute(st["qc"], **more)
    if kind == "mo":
        okgrid.set_grid(*st["axes"], is_vector=False)
        return core.rho_compute(st["qc"], calc_mo=True)
    if kind == "ao":
        okgrid.set_grid(*st["axes"], is_vector=False)
        return core.ao_creator(st["qc"].geo_spec, st["qc"].ao_spec)
    if kind == "fit":
        for p in st["params"]:
            p.grad = None
        rho, grad = st["model"](*st["params"])
        loss = density_fit_loss(rho, grad, st["target"][0], st["target"][1], st["weights"])
        loss.backward()
        return [loss.detach()] + [p.grad for p in st["params"]]
    if kind == "batch":
        st["batch"].run()
        return [[m["rho"], m["grad"]] for m in st["batch"].mols]
    if kind == "overlap":
        return [st["plan"].run(st["geo"], st["geo"], d) for d in range(4)]
    if kind == "detci":
        return [detci.rho(st["zero"], st["sing"], st["mo"], reference_slicing=False),
                detci.jab(st["zero"], st["sing"], st["mo"], st["drv"], reference_slicing=False)]
    raise ValueError(kind)


def work(case):
    """Grid values: coordinates read once, outputs written once; arithmetic: the products
    of MO coefficients and AO values (2 per channel) and one exponential and three
    operations per primitive and point, an AO value counted as ten operations."""
    kind = case["kind"]
    if kind in ("density", "mo", "ao"):
        n = _npts(case)
        nao, nmo = _ncart(case["atoms"], case["basis"]), _nmo(case["atoms"])
        heavy = _heavy(case["atoms"])
        nprim = heavy * (15 if case["basis"] == "cart" else 16) + 5 * (case["atoms"] - heavy)
        if kind == "ao":
            ch, out, mos = 1, _nao(case["atoms"], case["basis"]), 0
        elif kind == "mo":
            ch, out, mos = 1, nmo, nmo
        else:
            ch = {"rho": 1, "grad": 4, "laplacian": 7}[case["what"]]
            # (value and derivatives; the Laplacian call returns its three terms and their sum)
            out, mos = {"rho": 1, "grad": 4, "laplacian": 5}[case["what"]], nmo
        read = 24.0 * n if case["grid"] == "points" else 0.0
        return {"bytes": read + 8.0 * out * n + 8.0 * (nao * mos + 2 * nprim),
                "flops": n * (2.0 * ch * nao * mos + 4.0 * nprim + 10.0 * ch * nao)}
    if kind == "fit":
        n = case["nx"] * case["ny"] * case["nz"]
        nao, nmo = _nao(case["atoms"], "cart"), _nmo(case["atoms"])
        heavy = _heavy(case["atoms"])
        nprim = heavy * 15 + 5 * (case["atoms"] - heavy)
        # forward (4 channels), the same MOs again for the cotangents, C^T W, C^T V, W chi^T, V G^T
        return {"bytes": 8.0 * n * 5 + 16.0 * nao * nmo,
                "flops": n * (2.0 * (4 + 4 + 4) * nao * nmo + 20.0 * nprim + 140.0 * nao)}
    if kind == "batch":
        b = f = 0.0
        for i in range(case["molecules"]):
            span = case["max_atoms"] - case["min_atoms"]
            atoms = case["min_atoms"] + (i * span) // max(1, case["molecules"] - 1)
            n = atoms * case["radial"] * case["angular"]
            b += 56.0 * n
            f += n * (8.0 * _nao(atoms, "cart") * _nmo(atoms) + 40.0 * _nao(atoms, "cart"))
        return {"bytes": b, "flops": f}
    if kind == "overlap":
        nao = _nao(case["atoms"], case["basis"])
        heavy = _heavy(case["atoms"])
        # primitives times Cartesian components of each shell
        rows = heavy * (10 + 12 + 6 + (10 if case["basis"] == "sph" else 0)) + 7 * (case["atoms"] - heavy)
        return {"bytes": 4 * 8.0 * nao * nao, "flops": 4 * 10.0 * rows * rows}
    n, m = case["npts"], case["nmo"]
    return {"bytes": 8.0 * n * (4 * m + 4), "flops": n * (m * (m + 1.0) + 2.0 * m * m + 6.0 * m)}


# ------------------------------------------------------------------ exact values
_CART = [[(0, 0, 0)], [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
         [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)],
         [(3, 0, 0), (0, 3, 0), (0, 0, 3), (1, 2, 0), (2, 1, 0), (2, 0, 1), (1, 0, 2), (0, 1, 2), (0, 2, 1), (1, 1, 1)]]


def _real_harmonics(L):
    """Rows of real solid harmonics over the normalised Cartesian components, in the order
    m = 0, 1, -1, 2, -2, ... (p: 1, -1, 0)."""
    r = math.sqrt
    if L == 0:
        return numpy.eye(1)
    if L == 1:
        return numpy.eye(3)
    if L == 2:
        rows = [{(0, 0, 2): 1, (2, 0, 0): -0.5, (0, 2, 0): -0.5}, {(1, 0, 1): 1}, {(0, 1, 1): 1},
                {(2, 0, 0): r(3) / 2, (0, 2, 0): -r(3) / 2}, {(1, 1, 0): 1}]
    else:
        a, b, c = r(6 / 5.0), r(6) / 4, r(6 / 5.0) / 4
        rows = [{(0, 0, 3): 1, (2, 0, 1): -3 / (2 * r(5)), (0, 2, 1): -3 / (2 * r(5))},
                {(1, 0, 2): a, (3, 0, 0): -b, (1, 2, 0): -c}, {(0, 1, 2): a, (0, 3, 0): -b, (2, 1, 0): -c},
                {(2, 0, 1): r(3) / 2, (0, 2, 1): -r(3) / 2}, {(1, 1, 1): 1},
                {(3, 0, 0): r(10) / 4, (1, 2, 0): -3 * r(2) / 4}, {(0, 3, 0): -r(10) / 4, (2, 1, 0): 3 * r(2) / 4}]
    T = numpy.zeros((len(rows), len(_CART[L])))
    for i, row in enumerate(rows):
        for k, v in row.items():
            T[i, _CART[L].index(k)] = v
    return T


def _dfact(n):
    return 1 if n <= 0 else n * _dfact(n - 2)


def _shells(qc):
    """(atom, L, alpha, c, T) per shell; T maps Cartesian components to output rows."""
    out = []
    sph = bool(getattr(qc.ao_spec, "spherical", False))
    for s in qc.ao_spec:
        L = "spdf".index(s["type"])
        a = numpy.asarray(s["coeffs"], dtype=numpy.float64)
        T = _real_harmonics(L) if sph else numpy.eye(len(_CART[L]))
        out.append((int(s["atom"]), L, a[:, 0], a[:, 1], T))
    return out


def _ao_values(shells, geo, alpha, coef, pts, nch, spherical=True):
    """(nch, nao, n): values, then d/dx, d/dy, d/dz, then xx, yy, zz, of every AO at pts (3, n);
    geo, alpha and coef are tensors (differentiable)."""
    blocks, p0, last, memo = [], 0, -1, None
    for atom, L, a, _, T in shells:
        if atom != last:
            X = pts - geo[atom][:, None]
            rr, last = (X * X).sum(0), atom
            pw = [torch.ones_like(X), X]
        while len(pw) < L + 3:
            pw.append(pw[-1] * X)
        al, c = alpha[p0:p0 + len(a)], coef[p0:p0 + len(a)]
        p0 += len(a)
        w = c * (2.0 / math.pi) ** 0.75 * 2.0 ** L * al ** ((2.0 * L + 3.0) / 4.0)
        e = w[:, None] * torch.exp(-al[:, None] * rr[None])
        R = [e.sum(0)]
        if nch > 1:
            R.append((al[:, None] * e).sum(0))
        if nch > 4:
            R.append((al[:, None] ** 2 * e).sum(0))
        rows = []
        for lx in _CART[L]:
            f = [pw[n][d] for d, n in enumerate(lx)]
            g = 1.0 / math.sqrt(_dfact(2 * lx[0] - 1) * _dfact(2 * lx[1] - 1) * _dfact(2 * lx[2] - 1))
            vals = [f[0] * f[1] * f[2] * R[0]]
            for order in (1, 2)[: 0 if nch == 1 else 1 if nch == 4 else 2]:
                for d in range(3):
                    n = lx[d]
                    if order == 1:
                        t = -2.0 * pw[n + 1][d] * R[1]
                        if n:
                            t = t + n * pw[n - 1][d] * R[0]
                    else:
                        t = 4.0 * pw[n + 2][d] * R[2] - 2.0 * (2 * n + 1) * pw[n][d] * R[1]
                        if n > 1:
                            t = t + n * (n - 1) * pw[n - 2][d] * R[0]
                    u, v = [f[k] for k in range(3) if k != d]
                    vals.append(t * u * v)
            rows.append(g * torch.stack(vals))
        B = torch.stack(rows)  # (ncart, nch, n)
        if len(T) != len(rows) or not numpy.array_equal(T, numpy.eye(len(T))):
            B = torch.einsum("rc,chn->rhn", torch.as_tensor(T, dtype=B.dtype, device=B.device), B)
        blocks.append(B)
    return torch.cat(blocks).transpose(0, 1)


def _parameters(qc, dev):
    t = lambda a: torch.tensor(numpy.asarray(a), dtype=torch.float64, device=dev)
    sh = _shells(qc)
    return (sh, t(qc.geo_spec), t(numpy.concatenate([s[2] for s in sh])), t(numpy.concatenate([s[3] for s in sh])),
            t(qc.mo_spec.get_coeffs()), t(qc.mo_spec.get_occ()))


def _flat_points(axes, dev, i, j):
    x, y, z = (torch.tensor(a, dtype=torch.float64, device=dev) for a in axes)
    q = torch.arange(i, j, device=dev)
    return torch.stack([x[q // (len(y) * len(z))], y[(q // len(z)) % len(y)], z[q % len(z)]])


def _density(par, pts, nch):
    sh, geo, al, c, C, occ = par
    phi = C @ _ao_values(sh, geo, al, c, pts, nch)  # (nch, nmo, n)
    rho = (occ[:, None] * phi[0] ** 2).sum(0)
    out = [rho]
    if nch > 1:
        g = 2.0 * (occ[:, None] * phi[0] * phi[1:4]).sum(1)
        out.append(g)
    if nch > 4:
        out[1] = 2.0 * (occ[:, None] * (phi[0] * phi[4:7] + phi[1:4] ** 2)).sum(1)
    return out


def _promolecule(geo, axes, dev):
    """Target density and gradient: a sum of exponentials at the nuclei."""
    pts = _flat_points(axes, dev, 0, len(axes[0]) * len(axes[1]) * len(axes[2]))
    rho = torch.zeros(pts.shape[1], dtype=torch.float64, device=dev)
    grad = torch.zeros_like(pts)
    for A in numpy.asarray(geo):
        d = pts - torch.tensor(A, dtype=torch.float64, device=dev)[:, None]
        r = torch.sqrt((d * d).sum(0) + 1e-4)
        e = torch.exp(-1.5 * r)
        rho += e
        grad -= 1.5 * (e / r) * d
    return rho, grad


def _chunk(nch, nao):
    return max(512, int(2.0e9 / (8.0 * nch * nao * 4)))


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    if kind in ("density", "mo", "ao"):
        rng, qc = _molecule(case["atoms"], case["basis"], seed)
        par = _parameters(qc, dev)
        n = _npts(case)
        if case["grid"] == "points":
            P = torch.tensor(_points(case, rng, qc.geo_spec), dtype=torch.float64, device=dev)
            part, N = lambda i, j: P[:, i:j], (n,)
        else:
            axes = _axes(case)
            part, N = lambda i, j: _flat_points(axes, dev, i, j), (case["nx"], case["ny"], case["nz"])
        nch = {"rho": 1, "grad": 4, "laplacian": 7}[case["what"]] if kind == "density" else 1
        step, got = _chunk(nch, _ncart(case["atoms"], case["basis"])), []
        for i in range(0, n, step):
            pts = part(i, min(n, i + step))
            if kind == "density":
                got.append([v.cpu() for v in _density(par, pts, nch)])
            else:
                v = _ao_values(*par[:4], pts, 1)[0]
                got.append([(par[4] @ v if kind == "mo" else v).cpu()])
        out = [torch.cat([g[k] for g in got], dim=-1) for k in range(len(got[0]))]
        out = [v.reshape(tuple(v.shape[:-1]) + N) for v in out]
        if kind != "density" or case["what"] == "rho":
            return out[0]
        return (out[0], out[1], out[1].sum(0)) if case["what"] == "laplacian" else (out[0], out[1])
    if kind == "fit":
        _, qc = _molecule(case["atoms"], "cart", seed)
        axes = _axes(case)
        sh, geo, al, c, C, occ = _parameters(qc, dev)
        if case["precision"] == "fp32":  # the float32 parameters' values
            geo, al, c, C = (v.to(torch.float32).to(torch.float64) for v in (geo, al, c, C))
        leaves = [v.requires_grad_(True) for v in (C, al, c, geo)]
        rt, gt = _promolecule(qc.geo_spec, axes, dev)
        gen = torch.Generator(device=dev).manual_seed(seed)
        w = torch.rand(_npts(case), generator=gen, dtype=torch.float64, device=dev)
        total = torch.zeros((), dtype=torch.float64, device=dev)
        step = _chunk(4, 8 * _nao(case["atoms"], "cart"))
        for i in range(0, _npts(case), step):
            j = min(_npts(case), i + step)
            rho, grad = _density((sh, geo, al, c, C, occ), _flat_points(axes, dev, i, j), 4)
            loss = (w[i:j] * (rho - rt[i:j]) ** 2).sum() + 0.1 * ((grad - gt[:, i:j]) ** 2).sum()
            loss.backward()
            total += loss.detach()
        return [total] + [v.grad for v in leaves]
    if kind == "batch":
        got = []
        for i in range(case["molecules"]):
            span = case["max_atoms"] - case["min_atoms"]
            atoms = case["min_atoms"] + (i * span) // max(1, case["molecules"] - 1)
            _, qc = _molecule(atoms, "cart", [seed, i])
            par = _parameters(qc, dev)
            shell = (synthetic.becke_radial(case["radial"])[:, None, None] *
                     synthetic.fibonacci_sphere(case["angular"])[None]).reshape(-1, 3)
            P = torch.tensor((qc.geo_spec[:, None] + shell[None]).reshape(-1, 3).T.copy(), device=dev)
            step = _chunk(4, _nao(atoms, "cart"))
            parts = [_density(par, P[:, k:k + step], 4) for k in range(0, P.shape[1], step)]
            got.append([torch.cat([p[k] for p in parts], dim=-1) for k in range(2)])
        return got
    if kind == "overlap":
        return _exact_overlap(case, seed, dev)
    if kind == "detci":
        st = prepare(case, seed)
        M = torch.zeros((case["nmo"], case["nmo"]), dtype=torch.float64)
        F = torch.zeros_like(M)
        for cs, js in zip(*st["zero"]):
            for v, k in zip(cs, js):
                M[k, k] += v
        for v, (a, b) in zip(*st["sing"]):
            M[a, b] += v
            F[a, b] += v
        M, F, mo, drv = M.to(dev), F.to(dev), st["mo"], st["drv"]
        # j = -1/2 sum_ab F_ab (MO_a dMO_b - MO_b dMO_a)
        half = (F - F.T).T @ mo
        return [((M @ mo) * mo).sum(0), -0.5 * (half[None] * drv).sum(1)]
    return None


def _exact_overlap(case, seed, dev):
    """S and d/dx, d/dy, d/dz of the ket from the one-dimensional Gaussian product sums."""
    _, qc = _molecule(case["atoms"], case["basis"], seed)
    sh, geo, al, c, _, _ = _parameters(qc, dev)
    prim_row, l_row, norm, cart_of, T_blocks, k, p0 = [], [], [], [], [], 0, 0
    for atom, L, a, co, T in sh:
        for lx in _CART[L]:
            g = 1.0 / math.sqrt(_dfact(2 * lx[0] - 1) * _dfact(2 * lx[1] - 1) * _dfact(2 * lx[2] - 1))
            for q in range(len(a)):
                prim_row.append(p0 + q)
                l_row.append(lx)
                norm.append(g * co[q] * (2.0 / math.pi) ** 0.75 * 2.0 ** L * a[q] ** ((2.0 * L + 3.0) / 4.0))
                cart_of.append(k)
            k += 1
        p0 += len(a)
        T_blocks.append(torch.tensor(T, dtype=torch.float64, device=dev))
    ncart, top = k, max(s[1] for s in sh)
    atom_of = torch.tensor(numpy.concatenate([[s[0]] * len(s[2]) for s in sh]), device=dev)
    A = geo[atom_of]
    p = al[:, None] + al[None, :]
    inner = []  # one-dimensional overlaps s[d][a][b] over primitive pairs
    for d in range(3):
        AB = A[:, None, d] - A[None, :, d]
        PA, PB = -al[None, :] / p * AB, al[:, None] / p * AB
        s = [[None] * (top + 2) for _ in range(top + 1)]
        s[0][0] = torch.exp(-al[:, None] * al[None, :] / p * AB * AB) * torch.sqrt(math.pi / p)
        for a in range(top + 1):
            for b in range(top + 2):
                if a == 0 and b == 0:
                    continue
                if a > 0:
                    v = PA * s[a - 1][b]
                    if a > 1:
                        v = v + (a - 1) / (2 * p) * s[a - 2][b]
                    if b > 0:
                        v = v + b / (2 * p) * s[a - 1][b - 1]
                else:
                    v = PB * s[a][b - 1]
                    if b > 1:
                        v = v + (b - 1) / (2 * p) * s[a][b - 2]
                s[a][b] = v
        inner.append(s)
    rows = torch.tensor(prim_row, device=dev)
    lx = torch.tensor(l_row, device=dev)
    norm = torch.tensor(norm, dtype=torch.float64, device=dev)
    cart_of = torch.tensor(cart_of, device=dev)
    flat = [torch.stack([torch.stack([s[a][b] for b in range(top + 2)]) for a in range(top + 1)]) for s in inner]
    out = [torch.zeros((ncart, ncart), dtype=torch.float64, device=dev) for _ in range(4)]
    for i in range(0, len(rows), 256):
        r, l = rows[i:i + 256], lx[i:i + 256]

        def part(d, shift):
            b = lx[:, d] + shift
            v = flat[d][l[:, None, d], b.clamp(min=0)[None, :], r[:, None], rows[None, :]]
            return torch.where((b >= 0)[None, :], v, torch.zeros_like(v))

        plain = [part(d, 0) for d in range(3)]
        for o in range(4):
            f = list(plain)
            if o:
                d = o - 1
                f[d] = lx[None, :, d] * part(d, -1) - 2.0 * al[rows][None, :] * part(d, 1)
            v = f[0] * f[1] * f[2] * norm[i:i + 256, None] * norm[None, :]
            m = torch.zeros((len(r), ncart), dtype=torch.float64, device=dev).index_add_(1, cart_of, v)
            out[o].index_add_(0, cart_of[i:i + 256], m)
    T = torch.block_diag(*T_blocks)
    return [T @ S @ T.T for S in out]
