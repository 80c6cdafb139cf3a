"""Fock matrices of densities near the end of the double range: a power of two times those of the
density itself.

Tolerance: a sum of at most n^2 products in another order, n^2 2^-53 = 2e-13 at n = 43 (1e-12 asked)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units", [2, 3])
@pytest.mark.parametrize("power", [-900, 1000, 1009, 1012])
def test_powers_of_two(units, power):
    from pychem_gb300 import workloads
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    eng = GpuEngine(Molecule(workloads.alkane(units, seed=1), "6-31G")).prepare()
    eng.H = torch.zeros_like(eng.H)
    n = eng.nbf
    M = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(units))
    D = (M + M.T) / n
    s = 2.0 ** power
    for got, want in ((eng.fock(D * s), eng.fock(D)), (eng.fock_u(D * s, D * s)[1], eng.fock_u(D, D)[1]),
                      (eng.coulomb_exchange((D * s)[None])[1], eng.coulomb_exchange(D[None])[1])):
        assert float((got / s - want).abs().max()) < 1e-12 * float(want.abs().max())
