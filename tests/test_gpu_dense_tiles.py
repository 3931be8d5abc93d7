"""The dense entry points' tiles at their edges: odd and even function counts
(8- and 16-byte copies), matrices that start 8 bytes off a 16-byte boundary,
points that do not fill a tile, orbital counts around the tile widths and
beyond one tile, functions in an order that breaks shells apart, and angular
momenta to 7 -- against plain torch FP64 of the same formulas (relative
2-norm 1e-12: sums of at most 3000 terms in FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402
from oracle import oracle as O  # noqa: E402

TOL = 1e-12


def _rel(a, b):
    return float((a - b).norm() / b.norm().clamp(min=1e-300))


def _colmajor(rows, cols, seed, off=0):
    """rows x cols matrix stored column-major, its data `off` doubles into a buffer"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    buf = torch.randn(rows * cols + off, dtype=torch.float64, device="cuda", generator=g)
    return buf[off:].view(cols, rows).t()


@pytest.mark.parametrize("nbf,npts,nocc,off", [(1, 1, 1, 0), (17, 63, 8, 0), (48, 257, 9, 1), (64, 1000, 33, 0),
                                               (71, 300, 70, 1), (130, 513, 130, 0)])
def test_density_and_sigma(nbf, npts, nocc, off):
    phi, gx, gy, gz = (_colmajor(nbf, npts, k, off) for k in range(4))
    C = _colmajor(nbf, nocc, 7, off)
    occ = torch.linspace(0.1, 2.0, nocc, dtype=torch.float64, device="cuda")
    T = C.t() @ phi
    rho = (occ[:, None] * T * T).sum(0)
    grad = torch.stack([2 * (occ[:, None] * T * (C.t() @ q)).sum(0) for q in (gx, gy, gz)])
    r, g, s = A.compute_density_and_sigma(phi, gx, gy, gz, C, occ)
    assert _rel(r, rho) <= TOL and _rel(g, grad) <= TOL and _rel(s, (grad * grad).sum(0)) <= TOL
    assert _rel(A.compute_density(phi, C, occ), rho) <= TOL


@pytest.mark.parametrize("nbf,naux,npts,off", [(1, 1, 1, 0), (17, 33, 300, 0), (48, 143, 2500, 1), (70, 64, 129, 0)])
def test_coulomb(nbf, naux, npts, off):
    phi, Vw = _colmajor(nbf, npts, 1, off), _colmajor(naux, npts, 2, off)
    K = max(1, naux - 3)
    X, C = _colmajor(naux, K, 3), _colmajor(nbf, 5, 4)
    occ = torch.ones(5, dtype=torch.float64, device="cuda")
    v = Vw.t() @ (X @ (X.t() @ (Vw @ ((C.t() @ phi) ** 2).sum(0))))
    J = A.compute_coulomb(C, occ, phi, None, Vw, X)
    assert _rel(J, (phi * v) @ phi.t()) <= TOL


@pytest.mark.parametrize("npts", [1, 127, 300])
@pytest.mark.parametrize("order", ["shells", "shuffled"])
def test_collocation_and_potentials(npts, order):
    rng = np.random.default_rng(npts)
    funcs = [(l + 1 + k, l, m, 0.4 + 0.3 * l + 0.2 * k, *c) for c in rng.normal(size=(2, 3)) for l in range(8)
             for k in range(2) for m in range(-l, l + 1)]
    if order == "shuffled":
        funcs = [funcs[i] for i in rng.permutation(len(funcs))][:97]  # odd count, shells broken apart
    pts = 3 * rng.normal(size=(npts, 3))
    w = rng.uniform(0.1, 1.0, npts)
    b, ob = A.make_manual_basis(funcs), O.make_manual_basis(funcs)
    ref = O.collocation(ob, pts, grad=True)
    for a, r in zip(A.fill_grad_collocation(b, pts), ref):
        r = np.asarray(r)
        assert np.linalg.norm(a.cpu().numpy() - r) <= TOL * np.linalg.norm(r)
    assert np.linalg.norm(A.fill_collocation(b, pts).cpu().numpy() - ref[0]) <= TOL * np.linalg.norm(ref[0])
    Vw = A.sto_potential_collocation_scaled(b, pts, w).cpu().numpy()
    Vo = np.asarray(O.potential_collocation(ob, pts, w))
    assert np.linalg.norm(Vw - Vo) <= 1e-11 * np.linalg.norm(Vo)


@pytest.mark.parametrize("nspin,lda,npts", [(1, False, 101), (2, False, 130), (2, True, 1)])
def test_dense_xc(nspin, lda, npts):
    c, Z = M.water_cluster(2, seed=5)
    funcs = M.sto_basis(c, Z)[:-1]  # 95 functions
    g = A.make_flat_grid(c, Z, 20, 11, weight_threshold=1e-15, radial="ta")
    pts, w = g.quad_points[-npts:], g.weights[-npts:]
    b = A.make_manual_basis(funcs)
    Cs = [M.random_orbitals(len(funcs), 9, seed=s) for s in range(nspin)]
    occ = [np.ones(9)] * nspin
    xc = ("LDA_X", "LDA_C_VWN") if lda else ("GGA_X_PBE", "GGA_C_PBE")
    phi = A.fill_grad_collocation(b, pts)
    if lda:
        r = A.compute_lsda(phi[0], w, Cs[0], occ[0], Cs[1], occ[1], xc)
    elif nspin == 1:
        r = A.compute_gga(*phi, w, Cs[0], occ[0], xc)
    else:
        r = A.compute_gga_lsda(*phi, w, Cs[0], occ[0], Cs[1], occ[1], xc)
    Eo, Vo = O.xc_build(O.make_manual_basis(funcs), pts, w, [1, 7] if lda else [101, 130], Cs, occ)
    assert abs(r[0] - Eo) <= 1e-10 * max(abs(Eo), 1e-12)
    for V, Vr in zip(r[1:], Vo):
        assert np.abs(V.cpu().numpy() - Vr).max() <= 1e-10 * max(1.0, np.abs(Vr).max())
