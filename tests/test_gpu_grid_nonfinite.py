"""A grid with a NaN point must not give a finite answer: the point's batch
keeps its blocks (a NaN must not get into the box that they are screened
against), so the mixed build reports it and the FP64 matrices show it.  One
function block and several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import _lib as L  # noqa: E402
from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402

NKX_ERR_NUMERIC = 5


@pytest.mark.parametrize("n", [1, 3])
@pytest.mark.parametrize("axes", [slice(0, 3), slice(1, 2)])
def test_nan_point_is_reported(n, axes):
    c, Z = M.water_cluster(n, seed=n)
    funcs = M.sto_basis(c, Z)
    g = A.make_flat_grid(c, Z, 20, 11, weight_threshold=1e-15, radial="ta")
    pts = g.quad_points.copy()
    pts[len(pts) // 2, axes] = np.nan
    fb = A.FockBuilder(c, Z, A.make_manual_basis(funcs), (pts, g.weights))
    assert (fb.batch_blocks() > 0).all()
    Cm, occ = M.random_orbitals(len(funcs), 5, seed=0), np.ones(5)
    with pytest.raises(L.NkxError) as e:
        fb.build([Cm], [occ], precision="mixed")
    assert e.value.code == NKX_ERR_NUMERIC
    V = fb.build([Cm], [occ], precision="fp64")[1]
    assert not np.isfinite(V[0]).all()
    fb.close()
