"""The plan's J with aux functions that do not come in complete shells of l <= 3:
functions to l = 5, only l >= 4, shells without their m = 0, functions in
random order, s functions that overfill a group -- against the dense sequence
with the same half inverse (a random one: the fit then amplifies nothing).
FP64: sums of at most 1e4 terms, 1e-11 relative; mixed: FP32 radial factors,
6e-8 each, 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402


def _sets(c):
    full = [(l + 1, l, m, 0.8 * 1.6 ** k + 0.3 * l, *x) for x in c for l in range(6) for k in range(2)
            for m in range(-l, l + 1)]
    return {"to l = 5": full, "l >= 4": [f for f in full if f[1] >= 4],
            "no m = 0": [f for f in full if f[1] in (1, 2) and f[2] != 0],
            "random order": [full[i] for i in np.random.default_rng(0).permutation(len(full))],
            "many s": [(1, 0, 0, 0.3 * 1.3 ** k, *x) for x in c for k in range(20)]}


@pytest.mark.parametrize("name", ["to l = 5", "l >= 4", "no m = 0", "random order", "many s"])
def test_j_of_any_aux_set(name):
    c, Z = M.water()
    funcs = M.sto_basis(c, Z)
    aux = _sets(c)[name]
    b, ab = A.make_manual_basis(funcs), A.make_manual_basis(aux)
    g = A.make_flat_grid(c, Z, 30, 11, weight_threshold=1e-15, radial="ta")
    Cm, occ = M.random_orbitals(len(funcs), 5, seed=1), np.ones(5)
    X = np.random.default_rng(1).normal(size=(len(aux), 7))
    J = A.compute_coulomb(Cm, occ, A.fill_collocation(b, g.quad_points), None,
                          A.sto_potential_collocation_scaled(ab, g.quad_points, g.weights), X).cpu().numpy()
    fb = A.FockBuilder(c, Z, b, g, aux=ab)
    fb.set_half_inverse(X)
    for precision, tol in (("fp64", 1e-11), ("mixed", 1e-6)):
        got = fb.build([Cm], [occ], precision=precision, want_J=True)[2]
        assert np.linalg.norm(got - J) <= tol * np.linalg.norm(J)
    fb.close()
