"""Edges of the plan's choices: the FP64 V tile at 64 and 65 functions (the last
basis that fills two slots of its block and the first that does not), in the
build and in the core Hamiltonian; blocks sorted by reach, at two screening
tolerances; the mixed density on either side of its rule for few batches.  Oracle gates as for screened builds: FP64 1e-10 relative on E and
1e-11 absolute on V unscreened; the tolerance of the dropped terms otherwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402
from oracle import oracle as O  # noqa: E402

PBE = [101, 130]


@pytest.mark.parametrize("nbf", [63, 64, 65])
def test_v_tile_of_half_a_block(nbf):
    c, Z = M.water_cluster(2, seed=3)
    funcs = M.sto_basis(c, Z)[:nbf]
    b = A.make_manual_basis(funcs)
    g = A.make_flat_grid(c, Z, 20, 11, weight_threshold=1e-15, radial="ta")
    Cm, occ = M.random_orbitals(nbf, 7, seed=nbf), np.ones(7)
    fb = A.FockBuilder(c, Z, b, g)
    E, V, _ = fb.build([Cm], [occ], precision="fp64")
    Eo, Vo = O.xc_build(O.make_manual_basis(funcs), g.quad_points, g.weights, PBE, [Cm], [occ])
    assert abs(E - Eo) <= 1e-10 * abs(Eo) and np.abs(V[0] - Vo[0]).max() <= 1e-11
    dense = A.compute_core_hamiltonian(b, c, Z, g.quad_points, g.weights)
    for got, ref in zip(fb.core_hamiltonian(c, Z), dense):
        ref = ref.cpu().numpy()
        assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
    fb.close()


@pytest.mark.parametrize("tol", [1e-10, 1e-6])
def test_blocks_sorted_by_reach(tol, monkeypatch):
    # eight close centres, each with a far-reaching, a middle and a tight shell of
    # 16 functions: sorted by reach they are one block each, and the number of
    # significant (batch, block) pairs is that of this order and no other
    c = np.array([[0.6 * (k & 1), 0.6 * (k >> 1 & 1), 0.6 * (k >> 2)] for k in range(8)])
    Z, zetas = np.ones(8, np.int32), (0.6, 3.0, 15.0)
    funcs = [(l + 1, l, m, z, *x) for x in c for z in zetas for l in range(4) for m in range(-l, l + 1)]
    opts = A._opts

    def with_tol(*a, **k):
        o = opts(*a, **k)
        o.screen_tol = tol
        return o
    monkeypatch.setattr(A, "_opts", with_tol)
    # points all over a box that only the far-reaching functions fill
    pts, w = np.random.default_rng(0).uniform(-18.0, 18.0, (20000, 3)), np.full(20000, 0.5)
    fb = A.FockBuilder(c, Z, A.make_manual_basis(funcs), (pts, w))
    boxes = A.create_bounding_boxes(A.FlatGrid(pts.copy(), w.copy(), c, Z, None), 256).cpu().numpy()
    radii = A.cutoff_radii(A.make_manual_basis(funcs, 1e-6 * tol))
    zeta = np.array([f[3] for f in funcs])
    centre = np.array([f[4:] for f in funcs])
    gap = np.maximum(np.maximum(boxes[:, None, 0] - centre, centre - boxes[:, None, 1]), 0.0)
    near = np.linalg.norm(gap, axis=2) <= radii
    pairs = sum(int(near[:, zeta == z].any(axis=1).sum()) for z in zetas)
    assert fb.info()["npairs"] == pairs < 0.9 * 3 * len(boxes)
    Cm, occ = M.random_orbitals(len(funcs), 3, seed=1), np.ones(3)
    Eo, Vo = O.xc_build(O.make_manual_basis(funcs), pts, w, PBE, [Cm], [occ])
    for precision, e, v in (("fp64", 1e-10, 1e-10), ("mixed", 1e-6, 1e-7)):
        E, V, _ = fb.build([Cm], [occ], precision=precision)
        assert abs(E - Eo) <= max(e, tol) and np.abs(V[0] - Vo[0]).max() <= max(v, tol)
    fb.close()


@pytest.mark.parametrize("nbatch,nocc,nspin", [(1, 5, 1), (30, 16, 2), (40, 16, 2), (30, 40, 1), (40, 17, 1), (3, 65, 1)])
def test_mixed_density_of_few_batches(nbatch, nocc, nspin):
    c, Z = M.water_cluster(3, seed=5)
    funcs = M.sto_basis(c, Z)
    g = A.make_flat_grid(c, Z, 30, 17, weight_threshold=1e-15, radial="ta")
    pick = np.argsort(np.linalg.norm(g.quad_points - c.mean(0), axis=1))[:256 * nbatch - 7]
    pts, w = g.quad_points[pick], g.weights[pick]
    Cs = [M.random_orbitals(len(funcs), nocc, seed=s) for s in range(nspin)]
    occ = [np.linspace(1.0, 0.3, nocc)] * nspin
    fb = A.FockBuilder(c, Z, A.make_manual_basis(funcs), (pts, w))
    E, V, _ = fb.build(Cs, occ, precision="mixed")
    Eo, Vo = O.xc_build(O.make_manual_basis(funcs), pts, w, PBE, Cs, occ)
    assert abs(E - Eo) <= 1e-6 and max(np.abs(a - b).max() for a, b in zip(V, Vo)) <= 1e-7
    fb.close()
