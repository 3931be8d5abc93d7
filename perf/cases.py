"""Workloads that stand for what a user of the library has it do.

Each case is a dict of plain values; `kind` names the entry points it takes:

  build         FockBuilder.build, one SCF iteration's XC (+ grid DF-J) work
  gradient      FockBuilder.xc_gradient
  density       FockBuilder.density, rho / grad rho / sigma on the grid
  dense_xc      fill_grad_collocation + compute_gga(_lsda) / compute_lda / lsda
  dense_density compute_density_and_sigma on a collocation in hand
  dense_coulomb sto_potential_collocation_scaled + compute_coulomb
  becke         partition_becke_team on atom grids in hand

Molecules, bases and orbitals are the seeded synthetic ones of
nukexc_b200.molecules; grids are Treutler-Ahlrichs x Lebedev with Becke
weights.  Where an output has one entry per grid point the geometry belongs to
the case (the number of points with a weight above the threshold depends on
it) and the seed gives the orbitals.  `exact` restates the same quantities in plain torch FP64.
"""
import math

import numpy as np
import torch

from nukexc_b200 import api as A
from nukexc_b200 import molecules as M

F64 = torch.float64
FUNCS = {"lda": ("LDA_X", "LDA_C_VWN"), "pbe": ("GGA_X_PBE", "GGA_C_PBE"), "pbe_x": ("GGA_X_PBE",)}
LEBEDEV_POINTS = {11: 50, 17: 110, 23: 194, 29: 302}
# aux functions of the single-water SCF (91 per molecule)
SCF_AUX = {8: [(0, 6), (1, 5), (2, 4), (3, 2)], 1: [(0, 4), (1, 3), (2, 1)]}
HALF_INVERSE_THR = 1e-4
WEIGHT_THRESHOLD = 1e-15


# ------------------------------------------------------------------ cases --
def _build(n, functional="pbe", precision="mixed", nspin=1, mem="device", j="none", nrad=75, order=29, agg=False):
    return {"kind": "build", "n": n, "aggregate": agg, "functional": functional, "precision": precision,
            "nspin": nspin, "mem": mem, "j": j, "nrad": nrad, "order": order}


def listed():
    return [
        # one iteration of a small molecule's SCF with every matrix on the GPU: launches and latency
        dict(_build(1, functional="lda"), name="water_lda_mixed"),
        # the same molecule through a host driver in plain FP64, XC and separate J (SCF to 1e-8 Eh)
        dict(_build(1, functional="lda", precision="fp64", mem="host", j="separate"), name="water_lda_j_fp64"),
        # an ordinary cluster from a host SCF driver
        dict(_build(8, mem="host"), name="water8_pbe_mixed"),
        # open shell in FP64, a basis that does not fill its last function block
        dict(_build(5, precision="fp64", nspin=2), name="water5_pbe_open_fp64"),
        # XC and density-fitted Coulomb together
        dict(_build(8, j="separate"), name="water8_pbe_j_mixed"),
        # randomly packed C/H/N/O atoms in random order: uneven screening, many orbitals
        dict(_build(149, agg=True), name="aggregate149_pbe_mixed"),
        # the largest single-GPU cluster of the benchmark
        dict(_build(64), name="water64_pbe_mixed"),
        # forces in a geometry optimisation
        {"kind": "gradient", "n": 8, "functional": "pbe", "precision": "mixed", "nspin": 1, "nrad": 75, "order": 29,
         "name": "water8_gradient_mixed"},
        # the density on the grid for analysis, closed shell
        {"kind": "density", "n": 4, "nspin": 1, "grad": True, "nrad": 75, "order": 29, "name": "water4_density"},
        # the dense call sequence of a small molecule: collocation with gradients, then E and V
        {"kind": "dense_xc", "n": 1, "functional": "pbe", "nspin": 1, "nrad": 75, "order": 29,
         "name": "water_dense_gga"},
        # the dense Coulomb sequence: aux potentials on the grid, then J
        {"kind": "dense_coulomb", "n": 1, "nrad": 75, "order": 29, "name": "water_dense_coulomb"},
        # the Becke weights of a new geometry
        {"kind": "becke", "n": 16, "nrad": 75, "order": 29, "name": "water16_becke"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build"] * 7 + ["gradient", "density", "dense_xc", "dense_density", "dense_coulomb", "becke"])
    nrad, order = rng.randint(30, 75), rng.choice([17, 23, 29])
    if kind == "build":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        j = rng.choice(["none", "none", "separate", "fused"])
        nspin = rng.choice([1, 1, 2]) if j != "fused" else 1
        functional = rng.choice(["pbe", "pbe", "lda", "pbe_x"])
        mem = rng.choice(["device", "host"])
        if j == "none" and precision == "mixed" and rng.random() < 0.3:
            return _build(_log_int(rng, 12, 149), functional, precision, nspin, mem, j, nrad, order, True)
        top = 8 if j != "none" else 24 if precision == "mixed" else 12
        return _build(_log_int(rng, 1, top), functional, precision, nspin, mem, j, nrad, order)
    if kind == "gradient":
        return {"kind": kind, "n": _log_int(rng, 1, 8), "functional": rng.choice(["pbe", "lda"]),
                "precision": rng.choice(["mixed", "fp64"]), "nspin": rng.choice([1, 2]), "nrad": nrad, "order": order}
    if kind == "density":
        return {"kind": kind, "n": _log_int(rng, 1, 8), "nspin": rng.choice([1, 2]),
                "grad": rng.random() < 0.7, "nrad": nrad, "order": order}
    if kind == "dense_xc":
        return {"kind": kind, "n": rng.randint(1, 3), "functional": rng.choice(["pbe", "lda"]),
                "nspin": rng.choice([1, 2]), "nrad": nrad, "order": order}
    if kind == "becke":
        return {"kind": kind, "n": _log_int(rng, 1, 32), "nrad": nrad, "order": order}
    return {"kind": kind, "n": rng.randint(1, 3), "nrad": nrad, "order": order}


# ----------------------------------------------------------------- inputs --
def _molecule(case, seed):
    if case["kind"] in ("density", "dense_density", "dense_coulomb"):
        seed = 0  # per-point outputs: one geometry
    if case.get("aggregate"):
        c, Z = M.aggregate(case["n"], seed)
        return c, Z, M.aggregate_basis(c, Z), sum(Z) // 2
    if case["n"] == 1:
        # one water, turned at random so that each seed is another geometry
        c, Z = M.water_cluster(1, seed, jitter=0.0)
    else:
        c, Z = M.water_cluster(case["n"], seed)
    return c, Z, M.sto_basis(c, Z), 5 * case["n"]


def _aux_functions(case, c, Z):
    if case["kind"] == "build" and case["n"] == 1:
        return M.sto_basis(c, Z, SCF_AUX, alpha=0.8, beta=2.5)
    return M.aux_basis(c, Z)


def _orbitals(case, nbf, nocc, seed):
    """C and occupations per spin; the second spin has its last orbital empty."""
    ns = case.get("nspin", 1)
    Cs = [M.random_orbitals(nbf, nocc, 1000 * seed + s) for s in range(ns)]
    occ = [np.full(nocc, 2.0 if ns == 1 else 1.0) for _ in range(ns)]
    if ns == 2:
        occ[1][-1] = 0.0
    return Cs, occ


def _gpu(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=F64, device="cuda")


def prepare(case, seed):
    c, Z, funcs, nocc = _molecule(case, seed)
    st = {"case": case, "centers": c, "Z": Z}
    if case["kind"] == "becke":
        off, w, own = _atom_grids(case, Z)
        st.update(points=_gpu(c)[own] + off, weights=w, owner=own.to(torch.int32), centers=_gpu(c))
        return st
    grid = A.make_flat_grid(c, Z, case["nrad"], case["order"], weight_threshold=WEIGHT_THRESHOLD, radial="ta")
    basis = A.make_manual_basis(funcs)
    Cs, occ = _orbitals(case, len(funcs), nocc, seed)
    kind = case["kind"]
    if kind in ("build", "gradient", "density"):
        aux = A.make_manual_basis(_aux_functions(case, c, Z)) if case.get("j", "none") != "none" else None
        func = FUNCS[case.get("functional", "pbe")]
        st["fb"] = fb = A.FockBuilder(c, Z, basis, grid, aux=aux, func_ids=func)
        if aux is not None:
            # the fit with the thresholded half inverse, as the reference's driver does it
            fb.set_half_inverse(A.compute_half_inverse(fb.aux_metric(), HALF_INVERSE_THR).cpu().numpy())
        if case.get("mem") == "device":
            # orbitals as a device eigensolver leaves them
            Cs, occ = [_gpu(x) for x in Cs], [_gpu(x) for x in occ]
        st.update(C=Cs, occ=occ)
        return st
    st.update(basis=basis, points=_gpu(grid.quad_points), weights=_gpu(grid.weights), C=[_gpu(x) for x in Cs],
              occ=[_gpu(x) for x in occ])
    if kind == "dense_density":
        st["phi"] = A.fill_grad_collocation(basis, st["points"])
    if kind == "dense_coulomb":
        aux = A.make_manual_basis(_aux_functions(case, c, Z))
        S = A.coulomb_overlap_integral(aux, st["points"], st["weights"])
        st.update(aux=aux, X=A.compute_half_inverse(S, HALF_INVERSE_THR),
                  phi=A.fill_collocation(basis, st["points"]), phi_aux=A.fill_collocation(aux, st["points"]))
    return st


# -------------------------------------------------------------------- run --
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "becke":
        return {"weights": A.partition_becke_team(st["centers"], st["points"], st["owner"], st["weights"])}
    if kind == "build":
        E, V, J = st["fb"].build(st["C"], st["occ"], precision=case["precision"], want_J=case["j"] == "separate",
                                 fuse_j=case["j"] == "fused")
        out = {"E": E, "V": list(V)}
        if J is not None:
            out["J"] = J
        return out
    if kind == "gradient":
        return {"F": st["fb"].xc_gradient(st["C"], st["occ"], precision=case["precision"])}
    if kind == "density":
        r = st["fb"].density(st["C"], st["occ"], grad=case["grad"])
        return dict(zip(("rho", "grad", "sigma"), r)) if case["grad"] else {"rho": r}
    if kind == "dense_density":
        return dict(zip(("rho", "grad", "sigma"), A.compute_density_and_sigma(*st["phi"], st["C"][0], st["occ"][0])))
    if kind == "dense_coulomb":
        Vw = A.sto_potential_collocation_scaled(st["aux"], st["points"], st["weights"])
        return {"Vw": Vw, "J": A.compute_coulomb(st["C"][0], st["occ"][0], st["phi"], st["phi_aux"], Vw, st["X"])}
    # dense_xc
    func = FUNCS[case["functional"]]
    C, occ, w = st["C"], st["occ"], st["weights"]
    if case["functional"] == "lda":
        phi = A.fill_collocation(st["basis"], st["points"])
        r = A.compute_lda(phi, w, C[0], occ[0], func) if case["nspin"] == 1 else \
            A.compute_lsda(phi, w, C[0], occ[0], C[1], occ[1], func)
    else:
        phi = A.fill_grad_collocation(st["basis"], st["points"])
        r = A.compute_gga(*phi, w, C[0], occ[0], func) if case["nspin"] == 1 else \
            A.compute_gga_lsda(*phi, w, C[0], occ[0], C[1], occ[1], func)
    return {"E": r[0], "V": list(r[1:])}


# ------------------------------------------------------------------- work --
def _sizes(case):
    """(atoms, nbf, nocc, naux, points): points of the unpartitioned atom grids
    (a tenth of them, with a vanishing Becke weight, are dropped)."""
    n = case["n"]
    if case.get("aggregate"):
        nat = n
        h = n - 5 * (n // 10)  # about half hydrogen
        nbf, nocc, naux = 14 * (n - h) + 2 * h, int(0.5 * (6.6 * (n - h) + h)), 0
    else:
        nat, nbf, nocc = 3 * n, 48 * n, 5 * n
        naux = 91 if case["kind"] == "build" and n == 1 else 143 * n
    return nat, nbf, nocc, naux, nat * case["nrad"] * LEBEDEV_POINTS[case["order"]]


def work(case):
    nat, nbf, nocc, naux, npts = _sizes(case)
    kind, ns = case["kind"], case.get("nspin", 1)
    gga = case.get("functional", "pbe") != "lda"
    grid = 4 * 8 * npts  # points and weights once
    orb = 8 * ns * nbf * nocc
    colloc = npts * nbf * (30 if gga else 15)
    dens = 2 * npts * nbf * nocc * ns * (2 if gga else 1)  # value, and the gradient through Y = T0 C^T
    vmat = npts * nbf * nbf * ns * (2 if gga else 1)       # LDA's Phi diag(v) Phi^T is symmetric
    if kind == "becke":
        return {"bytes": 44 * npts, "flops": 40 * npts * min(nat, 12) ** 2}
    if kind == "build":
        by, fl = grid + orb + 8 * ns * nbf * nbf, colloc + dens + vmat
        if case["j"] != "none":
            fl += 4 * npts * naux
            by += 8 * naux * naux + (8 * nbf * nbf if case["j"] == "separate" else 0)
            fl += npts * nbf * nbf if case["j"] == "separate" else 0
        return {"bytes": by, "flops": fl}
    if kind == "gradient":
        return {"bytes": grid + orb + 24 * nat, "flops": 2 * colloc + 2 * dens + 40 * npts * min(nat, 12) ** 2}
    if kind == "density":
        return {"bytes": grid + orb + 8 * npts * ns * (5 if case["grad"] else 1), "flops": colloc + dens}
    if kind == "dense_density":
        return {"bytes": 4 * 8 * nbf * npts + orb + 8 * 5 * npts, "flops": dens}
    if kind == "dense_coulomb":
        # Vw written, read for y and for v; phi read for rho and J
        return {"bytes": grid + 8 * npts * (naux + nbf) + 8 * naux * naux,
                "flops": npts * (60 * naux + 4 * naux + 2 * nbf * nocc + nbf * nbf)}
    # dense_xc: the collocation matrices written by one call and read by the next
    return {"bytes": grid + orb + 2 * 8 * nbf * npts * (4 if gga else 1) + 8 * ns * nbf * nbf,
            "flops": colloc + dens + vmat}


# -------------------------------------------------------------- tolerance --
def tolerance(case):
    kind = case["kind"]
    if kind == "becke":
        # FP64 products of up to a dozen cell functions
        return {"rel": 1e-12, "max": 1e-10}
    mixed = case.get("precision") == "mixed"
    if kind == "gradient":
        # sums of large terms of both signs; 31-bit operands in the mixed form (3e-9 measured)
        return {"rel": 2e-8, "max": 1e-6} if mixed else {"rel": 1e-10, "max": 1e-8}
    if kind == "build" and mixed:
        # 31-bit operand rows: 4e-10 to 2e-8 measured against FP64, J (FP32 potentials) among it
        return {"rel": 8e-8, "max": 3e-6}
    # FP64 sums over 1e5 to 1e6 points in another order, 1e-15 to 1e-13 measured; the open-shell
    # functional and the J fit's threshold amplify them
    return {"rel": 1e-11, "max": 1e-9}


# ------------------------------------------------------------------ exact --
_LEBEDEV = {  # orbit representatives (a, b, c, weight), weights summing to 1
    17: [(0, 0, 1, 0.0038282704949371611), (0, 0.47836902881215021, 0.87815891060406615, 0.0096949963616630268),
         (0.18511563534473621, 0.18511563534473621, 0.96512403508659406, 0.0082117372831911097),
         (0.21595729184584844, 0.69042104838229224, 0.69042104838229224, 0.0099428148911781013),
         (0.39568947305594188, 0.39568947305594188, 0.82876998125259227, 0.0095954713360709605),
         (0.57735026918962573, 0.57735026918962573, 0.57735026918962573, 0.009793737512487511)],
    23: [(0, 0, 1, 0.001782340447244611), (0, 0.34577021976112832, 0.93831921813759156, 0.0050518460646148079),
         (0, 0.70710678118654757, 0.70710678118654757, 0.0057169059499771017),
         (0.12993354476500671, 0.12993354476500671, 0.98297230270725322, 0.0041067770281693937),
         (0.159041710538353, 0.52511857244364202, 0.83603601548245887, 0.0055302489162330944),
         (0.2892465627575439, 0.2892465627575439, 0.91250909686747372, 0.0051582377118053833),
         (0.31419699418258629, 0.67129734426952259, 0.67129734426952259, 0.0056087040825879972),
         (0.44469331787174371, 0.44469331787174371, 0.77749321931476711, 0.0055187714672736143),
         (0.57735026918962573, 0.57735026918962573, 0.57735026918962573, 0.0055733831788487374)],
    29: [(0, 0, 1, 0.00085459117251281483), (0, 0.26441528870606629, 0.96440891487920599, 0.0029823449631718041),
         (0, 0.57189558918789607, 0.82032641982775933, 0.0036008209322164601),
         (0.096183085226147838, 0.096183085226147838, 0.9907056213794081, 0.0023521014136891642),
         (0.1233548532583327, 0.41277240831685308, 0.90244252953300041, 0.0033923122050061698),
         (0.12923867271051442, 0.70117664160895454, 0.70117664160895454, 0.0036500458076772551),
         (0.22196452362941779, 0.22196452362941779, 0.94945431722644313, 0.0031089531224136749),
         (0.25100347517704652, 0.54486773725807736, 0.80007274940739515, 0.003571540554273387),
         (0.35156403455701052, 0.35156403455701052, 0.86764362454408339, 0.003449788424305883),
         (0.37103417838482095, 0.65663294102196124, 0.65663294102196124, 0.0036048226014198819),
         (0.47290541325810048, 0.47290541325810048, 0.74345204298755574, 0.003576729661743367),
         (0.57735026918962573, 0.57735026918962573, 0.57735026918962573, 0.0035991192850255709)],
}
_TA_XI = {1: 0.8, 6: 1.1, 7: 0.9, 8: 0.9}
BECKE_CLAMP = 5.0


def _lebedev(order):
    perms = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))
    pts, w = [], []
    for rep in _LEBEDEV[order]:
        own = []
        for p in perms:
            for s in range(8):
                q = tuple((-rep[p[k]] if s >> k & 1 else rep[p[k]]) + 0.0 for k in range(3))
                if q not in own:
                    own.append(q)
        pts += own
        w += [4 * math.pi * rep[3]] * len(own)
    return np.array(pts), np.array(w)


def _atom_grids(case, Z):
    """offsets from the owner, radial x angular weights and owners of every atom's points."""
    ang, aw = _lebedev(case["order"])
    n = case["nrad"]
    t = np.arange(1, n + 1) * math.pi / (n + 1)
    x = np.cos(t)
    off, w, own = [], [], []
    for a, z in enumerate(Z):
        s = _TA_XI[z] / math.log(2.0)
        lg = np.log(2.0 / (1.0 - x))
        r = s * (1.0 + x) ** 0.6 * lg
        dr = s * (0.6 * (1.0 + x) ** -0.4 * lg + (1.0 + x) ** 0.6 / (1.0 - x))
        rw = math.pi / (n + 1) * np.sin(t) * dr * r * r
        off.append((r[:, None, None] * ang[None]).reshape(-1, 3))
        w.append((rw[:, None] * aw[None]).reshape(-1))
        own.append(np.full(n * len(aw), a))
    return _gpu(np.concatenate(off)), _gpu(np.concatenate(w)), torch.as_tensor(np.concatenate(own), device="cuda")


def _becke(p, own, R):
    """P_owner / sum_i P_i of the clamped Becke cells at the points p."""
    n = R.shape[0]
    eye = torch.eye(n, dtype=F64, device=R.device)
    d = (R[:, None] - R[None] + eye[..., None]).norm(dim=-1).clamp(max=BECKE_CLAMP)
    r = (p[:, None] - R[None]).norm(dim=-1)
    Ps = []
    for i in range(n):
        f = ((r[:, i:i + 1] - r) / d[i]).clamp(-1.0, 1.0)
        for _ in range(3):
            f = f * (1.5 - 0.5 * f * f)
        s = 0.5 * (1.0 - f)
        Ps.append((s * (1 - eye[i]) + eye[i]).prod(dim=1))
    P = torch.stack(Ps, 1)
    return P.gather(1, own[:, None])[:, 0] / P.sum(1)


def _partitioned(p, w, own, R):
    step = max(1024, int(2e7) // len(R))
    return torch.cat([w[k:k + step] * _becke(p[k:k + step], own[k:k + step], R) for k in range(0, len(w), step)])


def _points(case, c, Z):
    off, w, own = _atom_grids(case, Z)
    R = _gpu(c)
    p = R[own] + off
    w = _partitioned(p, w, own, R)
    keep = w > WEIGHT_THRESHOLD
    return p[keep], w[keep]


def _harmonics(l, x, y, z):
    """(value, d/dx, d/dy, d/dz) of the real solid harmonics m = -l .. l."""
    pi, o = math.pi, torch.zeros_like(x)
    if l == 0:
        return [(o + math.sqrt(0.25 / pi), o, o, o)]
    if l == 1:
        k = math.sqrt(0.75 / pi)
        return [(k * y, o, o + k, o), (k * z, o, o, o + k), (k * x, o + k, o, o)]
    if l == 2:
        k, h, g = math.sqrt(15 / (4 * pi)), math.sqrt(15 / (16 * pi)), math.sqrt(5 / (16 * pi))
        return [(k * x * y, k * y, k * x, o), (k * y * z, o, k * z, k * y),
                (g * (2 * z * z - x * x - y * y), -2 * g * x, -2 * g * y, 4 * g * z),
                (k * x * z, k * z, o, k * x), (h * (x * x - y * y), 2 * h * x, -2 * h * y, o)]
    a, b, c = math.sqrt(35 / (32 * pi)), math.sqrt(105 / (4 * pi)), math.sqrt(21 / (32 * pi))
    d, e = math.sqrt(7 / (16 * pi)), math.sqrt(105 / (16 * pi))
    v = [a * (3 * x * x * y - y ** 3), b * x * y * z, c * y * (4 * z * z - x * x - y * y),
         d * z * (2 * z * z - 3 * x * x - 3 * y * y), c * x * (4 * z * z - x * x - y * y), e * z * (x * x - y * y),
         a * (x ** 3 - 3 * x * y * y)]
    return [(s, None, None, None) for s in v]  # l = 3: aux functions, values only


def _shells(funcs):
    """functions grouped by (n, l, m): list of (n, l, m, indices, zeta)."""
    by = {}
    for i, f in enumerate(funcs):
        by.setdefault(f[:3], []).append(i)
    return [(n, l, m, torch.as_tensor(ix, device="cuda"), _gpu([funcs[i][3] for i in ix]))
            for (n, l, m), ix in by.items()]


def _sto_norm(n, zeta):
    return (2 * zeta) ** (n + 0.5) / math.sqrt(math.factorial(2 * n))


def _collocation(shells, centers, p, grad):
    """[phi (, dx, dy, dz)], points x functions; centers: one row per function."""
    cols, order = [[] for _ in range(4 if grad else 1)], []
    for n, l, m, ix, zeta in shells:
        d = p[:, None] - centers[ix][None]
        x, y, z = d.unbind(-1)
        r = (d * d).sum(-1).sqrt()
        k = n - l - 1
        R = _sto_norm(n, zeta) * torch.exp(-zeta * r) * (r ** k if k else 1.0)
        S = _harmonics(l, x, y, z)[m + l]
        cols[0].append(R * S[0])
        if grad:
            q = S[0] * R * ((k / r if k else 0.0) - zeta) / r
            for t, u in enumerate((x, y, z)):
                cols[1 + t].append(R * S[1 + t] + q * u)
        order.append(ix)
    inv = torch.argsort(torch.cat(order))
    return [torch.cat(c, 1)[:, inv] for c in cols]


def _potentials(shells, centers, p):
    """electrostatic potentials of STOs, points x functions."""
    cols, order, radial = [], [], {}
    for n, l, m, ix, zeta in shells:
        d = p[:, None] - centers[ix][None]
        x, y, z = d.unbind(-1)
        r = (d * d).sum(-1).sqrt().clamp(min=1e-12)
        if m == -l:  # the shell's other functions follow in the same order
            t, a, b = zeta * r, n + l + 2, n - l + 1
            low = torch.special.gammainc(torch.full_like(t, a), t) * math.factorial(a - 1)
            up = torch.special.gammaincc(torch.full_like(t, b), t) * math.factorial(b - 1)
            radial[n, l] = (4 * math.pi / (2 * l + 1) * _sto_norm(n, zeta)
                            * (low / (zeta ** a * r ** (2 * l + 1)) + up / zeta ** b))
        cols.append(_harmonics(l, x, y, z)[m + l][0] * radial[n, l])
        order.append(ix)
    return torch.cat(cols, 1)[:, torch.argsort(torch.cat(order))]


def _pw92_g(rs, A0, a1, b1, b2, b3, b4):
    s = rs.sqrt()
    return -2 * A0 * (1 + a1 * rs) * torch.log1p(1 / (2 * A0 * (b1 * s + b2 * rs + b3 * rs * s + b4 * rs * rs)))


def _vwn_g(x, A0, b, c, x0):
    Q, X, X0 = math.sqrt(4 * c - b * b), x * x + b * x + c, x0 * x0 + b * x0 + c
    at = torch.atan(Q / (2 * x + b))
    return A0 * (torch.log(x * x / X) + 2 * b / Q * at
                 - b * x0 / X0 * (torch.log((x - x0) ** 2 / X) + 2 * (b + 2 * x0) / Q * at))


def _energy_density(functional, ra, rb, saa, sab, sbb):
    rho = ra + rb
    zeta, opz, omz = (ra - rb) / rho, 2 * ra / rho, 2 * rb / rho
    rs = (3 / (4 * math.pi * rho)) ** (1 / 3)
    fz = (opz ** (4 / 3) + omz ** (4 / 3) - 2) / (2 ** (4 / 3) - 2)
    z4 = zeta ** 4
    if functional == "lda":
        f = -0.75 * (6 / math.pi) ** (1 / 3) * (ra ** (4 / 3) + rb ** (4 / 3))
        x = rs.sqrt()
        eP = _vwn_g(x, 0.0310907, 3.72744, 12.9352, -0.10498)
        eF = _vwn_g(x, 0.01554535, 7.06042, 18.0578, -0.32500)
        eA = _vwn_g(x, -1 / (6 * math.pi ** 2), 1.13107, 13.0045, -0.0047584)
        fpp = 4 / (9 * (2 ** (1 / 3) - 1))
        return f + rho * (eP + eA * fz / fpp * (1 - z4) + (eF - eP) * fz * z4)

    def x_unpol(n, s2n):
        s2 = s2n / (4 * (3 * math.pi ** 2) ** (2 / 3) * n ** (8 / 3))
        return -0.75 * (3 / math.pi) ** (1 / 3) * n ** (4 / 3) * (1.804 - 0.804 / (1 + 0.2195149727645171 / 0.804 * s2))
    f = 0.5 * x_unpol(2 * ra, 4 * saa) + 0.5 * x_unpol(2 * rb, 4 * sbb)
    if functional == "pbe_x":
        return f
    gP = _pw92_g(rs, 0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294)
    gF = _pw92_g(rs, 0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517)
    gA = _pw92_g(rs, 0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671)
    ec = gP - gA * fz / 1.709920934161365617563962776245 * (1 - z4) + (gF - gP) * fz * z4
    beta, gamma = 0.06672455060314922, (1 - math.log(2)) / math.pi ** 2
    ph = 0.5 * (opz ** (2 / 3) + omz ** (2 / 3))
    ks2 = 4 * (3 * math.pi ** 2 * rho) ** (1 / 3) / math.pi
    t2 = (saa + 2 * sab + sbb) / (4 * ph * ph * ks2 * rho * rho)
    At2 = beta / gamma / torch.expm1(-ec / (gamma * ph ** 3)) * t2
    H = gamma * ph ** 3 * torch.log1p(beta / gamma * t2 * (1 + At2) / (1 + At2 + At2 * At2))
    return f + rho * (ec + H)


def _functional(functional, rho, grad):
    """energy density at rho (list per spin) and grad rho (list per spin of (points, 3) or None)."""
    ns = len(rho)
    ra, rb = (0.5 * rho[0], 0.5 * rho[0]) if ns == 1 else rho
    live = (ra + rb >= 1e-15)
    ra, rb = (torch.where(live, x.clamp(min=1e-30), torch.ones_like(x)) for x in (ra, rb))
    if grad is None:
        saa = sab = sbb = torch.zeros_like(ra)
    else:
        ga, gb = (0.5 * grad[0], 0.5 * grad[0]) if ns == 1 else grad
        saa, sab, sbb = ((u * v).sum(1) for u, v in ((ga, ga), (ga, gb), (gb, gb)))
        saa, sbb = saa.clamp(min=1e-40), sbb.clamp(min=1e-40)
    f = _energy_density(functional, ra, rb, saa, sab, sbb)
    return torch.where(live, f, torch.zeros_like(f))


def _density(phi, Cs, occ):
    rho, grad = [], []
    for C, o in zip(Cs, occ):
        T = phi[0] @ C
        rho.append((T * T) @ o)
        if len(phi) > 1:
            grad.append(torch.stack([2 * ((T * (q @ C)) @ o) for q in phi[1:]], 1))
    return rho, (grad if len(phi) > 1 else None)


def _chunks(n, nbf):
    step = max(256, int(1.5e7) // nbf)
    return [slice(k, min(n, k + step)) for k in range(0, n, step)]


def _half_inverse(S):
    D = S.diagonal().sqrt()
    lam, U = torch.linalg.eigh(S / (D[:, None] * D[None]))
    keep = lam.abs() > HALF_INVERSE_THR
    return U[:, keep] / lam.abs()[keep].sqrt() / D[:, None]


def _exact_v(functional, fn, centers, p, w, Cs, occ, aux, acenters):
    """E, V per spin, and with aux the Coulomb matrix."""
    nbf = len(centers)
    gga = functional != "lda"
    E, V = 0.0, [torch.zeros(nbf, nbf, dtype=F64, device="cuda") for _ in Cs]
    y = 0.0
    S = 0.0
    for s in _chunks(len(w), nbf):
        phi = _collocation(fn, centers, p[s], gga)
        rho, grad = _density(phi, Cs, occ)
        rho = [x.requires_grad_() for x in rho]
        grad = [x.requires_grad_() for x in grad] if gga else None
        f = _functional(functional, rho, grad)
        E += float((w[s] * f.detach()).sum())
        d = torch.autograd.grad(f.sum(), rho + (grad or []))
        for k in range(len(Cs)):
            z = 0.5 * d[k][:, None] * phi[0]
            if gga:
                for c in range(3):
                    z = z + d[len(Cs) + k][:, c:c + 1] * phi[1 + c]
            V[k] += phi[0].T @ (w[s][:, None] * z)
    V = [v + v.T for v in V]
    if aux is None:
        return E, V, None
    J = torch.zeros_like(V[0])
    for s in _chunks(len(w), max(nbf, len(acenters))):
        phi = _collocation(fn, centers, p[s], False)
        Vw = _potentials(aux, acenters, p[s]) * w[s][:, None]
        y = y + Vw.T @ sum(_density(phi, Cs, occ)[0])
        S = S + _collocation(aux, acenters, p[s], False)[0].T @ Vw
    X = _half_inverse(0.5 * (S + S.T))
    c = X @ (X.T @ y)
    for s in _chunks(len(w), max(nbf, len(acenters))):
        phi = _collocation(fn, centers, p[s], False)[0]
        v = (_potentials(aux, acenters, p[s]) @ c) * w[s]
        J += phi.T @ (v[:, None] * phi)
    return E, V, J


def exact(case, seed):
    c, Z, funcs, nocc = _molecule(case, seed)
    kind = case["kind"]
    functional = case.get("functional", "pbe")
    if kind == "gradient":
        return {"F": _exact_gradient(case, c, Z, funcs, nocc, seed)}
    if kind == "becke":
        off, w, own = _atom_grids(case, Z)
        return {"weights": _partitioned(_gpu(c)[own] + off, w, own, _gpu(c)).cpu().numpy()}
    p, w = _points(case, c, Z)
    fn, centers = _shells(funcs), _gpu([f[4:] for f in funcs])
    Cs, occ = ([_gpu(x) for x in xs] for xs in _orbitals(case, len(funcs), nocc, seed))
    if kind in ("density", "dense_density"):
        grad = case.get("grad", True)
        rows = [_density(_collocation(fn, centers, p[s], grad), Cs, occ) for s in _chunks(len(w), len(funcs))]
        rho = torch.stack([torch.cat([r[0][k] for r in rows]) for k in range(len(Cs))])
        if not grad:
            return {"rho": rho.cpu().numpy()}
        g = torch.stack([torch.cat([r[1][k] for r in rows]).T for k in range(len(Cs))])
        out = {"rho": rho, "grad": g, "sigma": (g * g).sum(1)}
        return {k: (v if kind == "density" else v[0]).cpu().numpy() for k, v in out.items()}
    want_j = kind == "dense_coulomb" or case.get("j", "none") != "none"
    afuncs = _aux_functions(case, c, Z) if want_j else []
    aux, acenters = (_shells(afuncs), _gpu([f[4:] for f in afuncs])) if want_j else (None, None)
    E, V, J = _exact_v("lda" if kind == "dense_coulomb" else functional, fn, centers, p, w, Cs, occ, aux, acenters)
    if kind == "dense_coulomb":
        Vw = _potentials(aux, acenters, p) * w[:, None]
        return {"Vw": Vw.T.cpu().numpy(), "J": J.cpu().numpy()}
    if case.get("j") == "fused":
        V, J = [v + J for v in V], None
    out = {"E": E, "V": [v.cpu().numpy() for v in V]}
    if J is not None:
        out["J"] = J.cpu().numpy()
    return out


def _exact_gradient(case, c, Z, funcs, nocc, seed):
    """dE_xc/dR by reverse-mode differentiation of the whole quadrature."""
    R = _gpu(c).requires_grad_()
    where = {tuple(x): i for i, x in enumerate(np.asarray(c))}
    atom = torch.as_tensor([where[tuple(f[4:])] for f in funcs], device="cuda")
    fn = _shells(funcs)
    Cs, occ = ([_gpu(x) for x in xs] for xs in _orbitals(case, len(funcs), nocc, seed))
    off, a, own = _atom_grids(case, Z)
    F = torch.zeros_like(R)
    for s in _chunks(len(a), 4 * max(len(funcs), len(Z) ** 2)):
        p = R[own[s]] + off[s]
        w = a[s] * _becke(p, own[s], R)
        keep = w.detach() > WEIGHT_THRESHOLD
        if not bool(keep.any()):
            continue
        p, w = p[keep], w[keep]
        phi = _collocation(fn, R[atom], p, case["functional"] != "lda")
        rho, grad = _density(phi, Cs, occ)
        F += torch.autograd.grad((w * _functional(case["functional"], rho, grad)).sum(), R)[0]
    return F.cpu().numpy()
