"""The mixed V contraction where its int32 sums are largest: 256 points in one
place, one p function there and weights that give every entry of both operand
rows one digit word, (-63, -128, -128, -128) (the largest 2^8 L2 + L3 there
is) or (64, -128, 127, 127) (the largest L2).  An overflow of a pair of levels
would be off by 2^32 in a sum of about 2^48.5 (1e-5); the digits' rounding is
2^-30 of the row maxima, hence 1e-8 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("word", [(-63, -128, -128, -128), (64, -128, 127, 127)])
def test_v_of_extreme_digit_words(word):
    X = ((word[0] * 256 + word[1]) * 256 + word[2]) * 256 + word[3]
    mant = X / 2.0 ** 30
    func = (2, 1, 0, 1.0, 0.0, 0.0, 0.0)  # p_z: phi has the sign of z
    b = O.make_manual_basis([func])
    phi_at = lambda z: float(np.asarray(O.collocation(b, np.array([[0.0, 0.0, z]]))).reshape(-1)[0])  # noqa: E731
    target = 0.125 * abs(mant)  # below the function's maximum
    lo, hi = 0.0, 0.9
    assert phi_at(hi) > target
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if phi_at(mid) < target else (lo, mid)
    z = float(np.sign(mant)) * hi
    phi = phi_at(z)
    assert abs(phi / 0.125 - mant) < 0.1 * 2.0 ** -30
    rho = torch.tensor([phi * phi], dtype=torch.float64, device="cuda")
    vrho = float(A.xc_eval("LDA_X", 1, rho)[1][0])
    w = mant / 8.0 / (0.5 * vrho * phi)  # Z = w vrho phi / 2 = mant / 8
    pts, ws = np.tile([[0.0, 0.0, z]], (256, 1)), np.full(256, w)
    fb = A.FockBuilder(np.zeros((1, 3)), np.ones(1, np.int32), A.make_manual_basis([func]), (pts, ws),
                       func_ids=("LDA_X",))
    V = {p: fb.build([np.ones((1, 1))], [np.ones(1)], precision=p)[1][0][0, 0] for p in ("fp64", "mixed")}
    fb.close()
    ref = 2 * 256 * phi * mant / 8.0
    assert abs(V["fp64"] - ref) <= 1e-12 * abs(ref)
    assert abs(V["mixed"] - ref) <= 1e-8 * abs(ref)
