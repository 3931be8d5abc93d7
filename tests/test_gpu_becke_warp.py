"""Becke weights where the warps' atom lists can go wrong: fewer atoms than warps,
lists of about 32 atoms, the last size of four warps and of eight, more atoms
than the lists hold (the per-thread path), the unclamped original, points far outside, and owners that
change inside a warp -- against the oracle's full loops (1e-13 absolute on
weights of at most 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("natoms,box,clamp", [(1, 3.0, 5.0), (2, 3.0, 0.0), (32, 9.0, 5.0), (33, 9.0, 0.0),
                                              (70, 30.0, 5.0), (144, 6.0, 5.0), (150, 6.0, 5.0), (150, 6.0, 0.0),
                                              (200, 40.0, 2.0), (96, 12.0, 5.0), (97, 12.0, 5.0), (400, 25.0, 5.0), (401, 25.0, 5.0)])
def test_becke_matches_oracle(natoms, box, clamp):
    rng = np.random.default_rng(natoms)
    c = rng.uniform(0, box, size=(natoms, 3))
    npts = 101 if natoms > 100 else 333
    own = rng.integers(0, natoms, npts).astype(np.int32)
    own[:64] = 0  # a warp with one owner, and one point far outside
    pts = c[own] + rng.normal(size=(npts, 3)) * rng.choice([0.1, 1.0, 4.0], size=(npts, 1))
    pts[5] += 60.0
    w = rng.uniform(0.5, 1.0, npts)
    got = A.partition_becke_team(c, pts, own, w, clamp=clamp).cpu().numpy()
    ref = O.becke(c, pts, own, w, clamp_R=clamp)
    assert np.abs(got - ref).max() <= 1e-13
