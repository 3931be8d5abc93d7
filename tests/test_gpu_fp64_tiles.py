"""The FP64 build's tiles at their edges: orbital tiles of 8 to 64 columns
(one and several of them), bases of a part of one function block, of one and
of several, closed and open shell, grids of one batch and more -- against the
oracle's dense build of the same grid (1e-10 relative on E, 1e-11 absolute
on V: FP64 sums of up to 1e4 points, whose terms are below 10)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("n,nocc,nspin,lda,npts", [
    (1, 1, 1, True, 200), (1, 8, 1, False, None), (1, 9, 2, True, 257), (1, 33, 1, False, 700),
    (3, 40, 2, False, None), (3, 64, 1, True, None), (3, 65, 1, False, 1500), (6, 130, 1, False, 2000)])
def test_fp64_build_matches_oracle(n, nocc, nspin, lda, npts):
    c, Z = M.water_cluster(n, seed=n)
    funcs = M.sto_basis(c, Z)
    g = A.make_flat_grid(c, Z, 20, 11, weight_threshold=1e-15, radial="ta")
    pick = slice(None) if npts is None else np.random.default_rng(0).permutation(len(g.weights))[:npts]
    pts, w = g.quad_points[pick], g.weights[pick]
    Cs = [M.random_orbitals(len(funcs), nocc, seed=s) for s in range(nspin)]
    occ = [np.linspace(1.0, 0.2, nocc) for _ in range(nspin)]
    xc = ("LDA_X", "LDA_C_VWN") if lda else ("GGA_X_PBE", "GGA_C_PBE")
    fb = A.FockBuilder(c, Z, A.make_manual_basis(funcs), (pts, w), func_ids=xc)
    E, V, _ = fb.build(Cs, occ, precision="fp64")
    E2, V2, _ = fb.build(Cs, occ, precision="fp64")
    Eo, Vo = O.xc_build(O.make_manual_basis(funcs), pts, w, [1, 7] if lda else [101, 130], Cs, occ)
    assert abs(E - Eo) <= 1e-10 * abs(Eo)
    for s in range(nspin):
        assert np.abs(V[s] - Vo[s]).max() <= 1e-11
    # the split sums are ordered: only rho's atomics over three and more orbital tiles may move the last bits
    assert all(np.abs(a - b).max() <= (0.0 if nocc <= 128 else 1e-13) for a, b in zip(V, V2))
    fb.close()
