"""Builds replayed from a CUDA graph with nuclear gradients in between.  The
mixed gradient shares the orbital-value and digit buffers of the mixed build
and needs larger ones: the graphs that hold the smaller ones must be dropped
before these are freed, so the first build after such a gradient is an ordinary
one (graph_replays unchanged), the next one is recorded again, and a later
gradient, which finds its buffers, leaves the graphs alone.  Builds equal those
of a plan without graphs (up to the order of atomic FP64 additions: 1e-12)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402
from nukexc_b200 import molecules as M  # noqa: E402


def _plan(xc, ypath, graph):
    c, Z = M.water_cluster(2, seed=4)
    g = A.make_flat_grid(c, Z, 30, 11, weight_threshold=1e-15, radial="ta")
    fb = A.FockBuilder(c, Z, A.make_manual_basis(M.sto_basis(c, Z)), g, func_ids=xc)
    fb.set_tuning(ypath=ypath)  # 1: the density gradient through Y, whose digits of T0 the gradient replaces too
    fb.set_graph(graph)
    return fb


@pytest.mark.parametrize("gradient", ["mixed", "fp64"])
@pytest.mark.parametrize("xc,ypath", [(("GGA_X_PBE", "GGA_C_PBE"), -1), (("GGA_X_PBE", "GGA_C_PBE"), 1),
                                      (("LDA_X", "LDA_C_VWN"), -1)])
def test_gradient_between_replays(xc, ypath, gradient):
    ref, fb = _plan(xc, ypath, False), _plan(xc, ypath, True)
    Cm = torch.as_tensor(M.random_orbitals(ref.nbf, 10, seed=5), device="cuda")
    occ = torch.full((10,), 2.0, dtype=torch.float64, device="cuda")
    Fr = ref.xc_gradient([Cm.cpu().numpy()], [occ.cpu().numpy()], precision=gradient)
    replays = 0

    def build(scale, step):
        nonlocal replays
        Ck = (Cm * scale).contiguous()
        E, V, _ = fb.build([Ck], [occ], precision="mixed")
        Eo, Vo, _ = ref.build([Ck], [occ], precision="mixed")
        assert abs(E - Eo) <= 1e-12 * abs(Eo)
        assert float((V[0] - Vo[0]).abs().max()) <= 1e-12 * float(Vo[0].abs().max())
        replays += step
        assert fb.info()["graph_replays"] == replays

    def grad():
        F = fb.xc_gradient([Cm.cpu().numpy()], [occ.cpu().numpy()], precision=gradient)
        assert abs(F - Fr).max() <= 1e-10 * max(1.0, abs(Fr).max())  # sums of 1e5 terms in varying order

    build(1.0, 0)
    build(1.001, 1)
    build(1.002, 1)
    grad()
    if gradient == "mixed":
        build(1.003, 0)  # its buffers have gone: an ordinary build
    build(1.004, 1)
    grad()
    build(1.005, 1)
    ref.close()
    fb.close()
