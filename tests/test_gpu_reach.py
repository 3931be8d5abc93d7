"""Function blocks grouped by reach: a chain of diffuse functions with tight ones
on its middle atoms, where grouping pays, gives the oracle's dense build (every
function on every point) within the gates of a screened build (FP64: 1e-10 on
E and V; mixed: 1e-6 and 1e-7); the density and the gradient follow the same
order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("nd", [1, 2])
def test_grouped_blocks_match_oracle(nd):
    c, Z = np.array([[0.0, 0.3 * i, 8.0 * i] for i in range(6)]), np.ones(6, np.int32)
    funcs = []
    for a in range(6):
        zetas = [0.5, 0.8][:nd] + ([6.0, 8.0, 11.0, 15.0] if a in (2, 3) else [])
        funcs += [(l + 1, l, m, z, *c[a]) for z in zetas for l in range(4 if z > 1 else 3) for m in range(-l, l + 1)]
    g = A.make_flat_grid(c, Z, 24, 11, weight_threshold=1e-15, radial="ta")
    Cm, occ = M.random_orbitals(len(funcs), 3, seed=1), np.ones(3)
    fb = A.FockBuilder(c, Z, A.make_manual_basis(funcs), g)
    E, V, _ = fb.build([Cm], [occ], precision="fp64")
    Em, Vm, _ = fb.build([Cm], [occ], precision="mixed")
    Eo, Vo, rho = O.xc_build(O.make_manual_basis(funcs), g.quad_points, g.weights, [101, 130], [Cm], [occ],
                             want_rho=True)
    assert abs(E - Eo) <= 1e-10 * abs(Eo) and np.abs(V[0] - Vo[0]).max() <= 1e-10
    assert abs(Em - Eo) <= 1e-6 and np.abs(Vm[0] - Vo[0]).max() <= 1e-7
    r = fb.density([Cm], [occ])[0]
    assert np.abs(r - np.asarray(rho).reshape(-1)[:len(r)]).max() <= 1e-10 * np.abs(r).max()
    F, Fm = (fb.xc_gradient([Cm], [occ], precision=p) for p in ("fp64", "mixed"))
    assert np.abs(F - Fm).max() <= 1e-6 and np.abs(F.sum(0)).max() <= 1e-9 * max(1.0, np.abs(F).max())
    i = fb.info()
    # the tight block is screened out towards the ends; in the order of the centres none is
    assert i["npairs"] < 0.95 * i["nbatches"] * i["nblocks"]
    fb.close()
