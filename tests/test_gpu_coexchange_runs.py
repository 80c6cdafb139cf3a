"""Co-densities whose quartets are many enough for threads to take several in a row: the digestion
against the products with pair matrices.

Tolerance: both sum at most n^2 products an element, magnitudes up to 30: n^2 2^-53 * 30 < 5e-11 (the
bar of test_gpu_coexchange.py)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system,basis", [("water4", "6-31G"), ("water4", "STO-3G"), ("alkane3", "cc-pVDZ")])
@pytest.mark.parametrize("nd", [1, 3, 15, 40])
def test_digestion_against_products(system, basis, nd, monkeypatch):
    from pychem_gb300 import engine, workloads
    from pychem_gb300.molecule import Molecule
    coords = workloads.water_cluster(nx=2, ny=2, nz=1, seed=3) if system == "water4" else workloads.alkane(3, seed=3)
    eng = engine.GpuEngine(Molecule(coords, basis)).prepare()
    n = eng.nbf
    W = 0.05 * torch.randn(nd, n, n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(nd))
    monkeypatch.setattr(engine, "COEXCHANGE_MIN", 10 ** 9)
    J, K = eng.coulomb_exchange(W)
    monkeypatch.setattr(engine, "COEXCHANGE_MIN", 1)
    Jp, Kp = eng.coulomb_exchange(W)
    assert float((J - Jp).abs().max()) < 5e-11 and float((K - Kp).abs().max()) < 5e-11
