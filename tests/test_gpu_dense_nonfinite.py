"""Infinite collocation values in the dense density: the orbitals that fill a
tile up must not turn the point's infinite density into NaN, which the
functionals skip.  Orbital counts that leave a tile partly filled."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402


@pytest.mark.parametrize("nocc", [1, 8, 9, 33, 65])
def test_infinite_value_gives_infinite_density(nocc):
    nbf, npts = 40, 300
    gen = torch.Generator(device="cuda").manual_seed(nocc)
    phi, gx, gy, gz = (torch.rand(npts, nbf, dtype=torch.float64, device="cuda", generator=gen).t() for _ in range(4))
    C = torch.rand(nocc, nbf, dtype=torch.float64, device="cuda", generator=gen).t() + 0.1
    occ = torch.ones(nocc, dtype=torch.float64, device="cuda")
    phi[3, 70] = float("inf")
    rho = ((C.t() @ phi) ** 2).sum(0)
    for got in (A.compute_density(phi, C, occ), A.compute_density_and_sigma(phi, gx, gy, gz, C, occ)[0]):
        assert torch.isinf(got[70]) and float(rho[70]) == float(got[70])
        ok = torch.arange(npts, device="cuda") != 70
        assert float((got - rho)[ok].abs().max()) <= 1e-12 * float(rho[ok].max())
