"""Becke weights of inputs that no grid should hold.  An owner outside
[0, natoms) owns nothing: weight 0.  A point with a NaN or infinite coordinate
has no weight: NaN, so that a build on it reports the point.  The other points
of the same warp keep their weights.  Sizes of each path: a thread
per point for few atoms, four warps, eight, and a thread per point for many; with
the clamp and without.  The first sizes of four warps also against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from oracle import oracle as O  # noqa: E402

SIZES = [3, 6, 97, 401]


def _case(natoms):
    rng = np.random.default_rng(natoms)
    c = rng.uniform(0, 3.0 * natoms ** (1 / 3), size=(natoms, 3))
    own = rng.integers(0, natoms, 70).astype(np.int32)
    return c, own, c[own] + rng.normal(size=(70, 3)), rng.uniform(0.5, 1.0, 70)


def _weights(c, pts, own, w, clamp):
    return A.partition_becke_team(c, pts, own, w, clamp=clamp).cpu().numpy()


@pytest.mark.parametrize("clamp", [5.0, 0.0])
@pytest.mark.parametrize("natoms", SIZES)
def test_owner_of_no_atom_has_no_weight(natoms, clamp):
    c, own, pts, w = _case(natoms)
    ref = _weights(c, pts, own, w, clamp)
    own[[1, 33, 64]] = -1, natoms, np.iinfo(np.int32).max
    got = _weights(c, pts, own, w, clamp)
    bad = np.isin(np.arange(70), [1, 33, 64])
    assert (got[bad] == 0.0).all() and (got[~bad] == ref[~bad]).all()


@pytest.mark.parametrize("clamp", [5.0, 0.0])
@pytest.mark.parametrize("natoms", SIZES)
def test_point_without_a_place_has_no_finite_weight(natoms, clamp):
    c, own, pts, w = _case(natoms)
    ref = _weights(c, pts, own, w, clamp)
    pts[2, 1], pts[40], pts[65, 0] = np.nan, np.nan, np.inf
    got = _weights(c, pts, own, w, clamp)
    bad = np.isin(np.arange(70), [2, 40, 65])
    assert np.isnan(got[bad]).all() and (got[~bad] == ref[~bad]).all()


@pytest.mark.parametrize("clamp", [5.0, 0.0])
@pytest.mark.parametrize("natoms", [5, 6, 7])
def test_first_sizes_of_four_warps(natoms, clamp):
    c, own, pts, w = _case(natoms)
    assert np.abs(_weights(c, pts, own, w, clamp) - O.becke(c, pts, own, w, clamp_R=clamp)).max() <= 1e-13
