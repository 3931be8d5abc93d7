"""Device memory between calls.  The dense entry points keep at most 256 MiB of
their workspace, which a plan counts as free and an allocation that needs it
gets; the FP64 gradient makes do with smaller pieces when the card is
nearly full.  The card is filled by one allocation that leaves a few hundred
MiB, which is what the calls below then have."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402

MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _card_with(free):
    filler = torch.empty(_free() - free, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()


def _dense_lda(nbf, npts):
    """an LDA build whose Z takes 8 nbf npts bytes of workspace, and what it
    took from the free memory when it returned"""
    phi = torch.rand(npts, nbf, dtype=torch.float64, device="cuda").t()
    C = torch.rand(3, nbf, dtype=torch.float64, device="cuda").t()
    w, occ = torch.ones(npts, dtype=torch.float64, device="cuda"), torch.ones(3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    A.compute_lda(phi, w, C, occ)
    return before - torch.cuda.mem_get_info()[0]  # no synchronisation in between


def test_dense_calls_keep_a_bounded_workspace():
    _dense_lda(16, 1000)  # kernels loaded
    assert _dense_lda(128, 1 << 20) <= (256 + 32) * MB  # 1 GiB of workspace


def _water(n, nrad, order, **kw):
    c, Z = M.water_cluster(n, seed=n)
    funcs = M.sto_basis(c, Z)
    g = A.make_flat_grid(c, Z, nrad, order, weight_threshold=1e-15, radial="ta")
    plan = lambda: A.FockBuilder(c, Z, A.make_manual_basis(funcs), g, **kw)  # noqa: E731
    return plan, M.random_orbitals(len(funcs), 5 * n, seed=1), np.ones(5 * n)


def test_plan_counts_kept_workspace_as_free():
    plan, _, _ = _water(1, 20, 11)
    plan().close()
    with _card_with(3 << 30):
        _dense_lda(128, 200 << 10)  # 192 to 256 MiB are kept
        free = _free()
        fb = plan()
        pairs = fb.tuning()["chunk_pairs"]  # a third of the free memory, 2 MiB a pair
        fb.close()
    assert (free + 170 * MB) / (6 * MB) <= pairs <= (free + 256 * MB) / (6 * MB)  # the plan has a few MiB already


def test_kept_workspace_goes_to_a_mixed_build():
    plan, Cm, occ = _water(4, 75, 29, workspace_bytes=800 * MB)  # 400 pairs: 0.41 GB of digits
    ref = plan()
    E0 = ref.build([Cm], [occ], precision="mixed")[0]
    ref.close()
    fb = plan()
    assert fb.info()["npairs"] >= 400
    _dense_lda(128, 200 << 10)  # 200 MiB of workspace are kept
    with _card_with(320 * MB):
        E = fb.build([Cm], [occ], precision="mixed")[0]
    assert abs(E - E0) <= 1e-12 * abs(E0)
    fb.close()


def test_fp64_gradient_on_a_nearly_full_card():
    plan, Cm, occ = _water(4, 75, 29)  # X of all pairs in one piece: 2 GB
    ref = plan()
    F0 = ref.xc_gradient([Cm], [occ])
    ref.close()
    fb = plan()
    with _card_with(700 * MB):
        F = fb.xc_gradient([Cm], [occ])
    assert np.abs(F - F0).max() <= 1e-11 * np.abs(F0).max()
    fb.close()
