"""The nuclear gradient's tiles at their edges: orbital counts around the
16-orbital step of X and beyond one density tile, a block with few functions,
one atom in a molecule of one, both spins, both precisions -- the derivative
along a random direction against Richardson-extrapolated central differences
of the GPU's own FP64 E_xc (steps 2e-3 and 1e-3 bohr: truncation h^4 of the
fifth derivatives, below 1e-7 of the terms, hence 2e-7 absolute per unit
direction; rounding 1e-13 / 1e-3)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402


@pytest.mark.parametrize("n,nocc,nspin,lda", [(1, 1, 1, False), (1, 16, 2, False), (2, 17, 1, True), (2, 65, 1, False),
                                              (4, 20, 2, False)])
def test_gradient_along_a_direction(n, nocc, nspin, lda):
    c, Z = M.water_cluster(n, seed=3 + n)
    xc = ("LDA_X", "LDA_C_VWN") if lda else ("GGA_X_PBE", "GGA_C_PBE")
    nbf = len(M.sto_basis(c, Z))
    Cs = [M.random_orbitals(nbf, nocc, seed=s) for s in range(nspin)]
    occ = [np.linspace(1.0, 0.3, nocc) for _ in range(nspin)]

    def plan(x):
        g = A.make_flat_grid(x, Z, 40, 17, weight_threshold=-1.0, radial="ta")  # every point, so none comes or goes
        return A.FockBuilder(x, Z, A.make_manual_basis(M.sto_basis(x, Z)), g, func_ids=xc)

    def energy(x):
        fb = plan(x)
        E = fb.build(Cs, occ, precision="fp64")[0]
        fb.close()
        return E
    d = np.random.default_rng(n).normal(size=c.shape)
    d /= np.linalg.norm(d)
    fd = [(energy(c + h * d) - energy(c - h * d)) / (2 * h) for h in (2e-3, 1e-3)]
    ref = (4 * fd[1] - fd[0]) / 3
    fb = plan(c)
    for precision, tol in (("fp64", 2e-7), ("mixed", 1e-6)):
        F = fb.xc_gradient(Cs, occ, precision=precision)
        assert abs((F * d).sum() - ref) <= tol
        assert np.abs(F.sum(0)).max() <= 1e-9 * max(1.0, np.abs(F).max())
    fb.close()


# the last and first sizes of four warps, of eight and of a thread per point for
# the weights' term; one s function an atom, the bounds of the test above
@pytest.mark.parametrize("natoms", [3, 48, 49, 192, 193])
def test_weight_term_along_a_direction(natoms):
    rng = np.random.default_rng(natoms)
    c = 2.4 * np.array([[i % 6, i // 6 % 6, i // 36] for i in range(natoms)]) + rng.uniform(-0.3, 0.3, (natoms, 3))
    Z, Cm, occ = np.ones(natoms, np.int32), M.random_orbitals(natoms, 2, seed=1), np.ones(2)

    def plan(x):
        g = A.make_flat_grid(x, Z, 20, 11, weight_threshold=-1.0, radial="ta")
        return A.FockBuilder(x, Z, A.make_manual_basis([(1, 0, 0, 1.1, *r) for r in x]), g)

    def energy(x):
        fb = plan(x)
        E = fb.build([Cm], [occ], precision="fp64")[0]
        fb.close()
        return E
    d = rng.normal(size=c.shape)
    d /= np.linalg.norm(d)
    fd = [(energy(c + h * d) - energy(c - h * d)) / (2 * h) for h in (2e-3, 1e-3)]
    fb = plan(c)
    F = fb.xc_gradient([Cm], [occ])
    fb.close()
    assert abs((F * d).sum() - (4 * fd[1] - fd[0]) / 3) <= 2e-7
    assert np.abs(F.sum(0)).max() <= 1e-9 * max(1.0, np.abs(F).max())
