"""Fock digestion over all lists in one call -- one shared launch below 304,000 quartets, one a
class above, several consecutive quartets a thread in long lists -- against the dense Coulomb
and exchange contractions.

Tolerance: F is a sum of up to n^2 (12,000) products of |D| <= 1 with integrals of total
magnitude below 1e3 an element; 2^-53 * sqrt(12000) * 1e3 = 1.2e-11 at most (2e-11 asked).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _coords(name):
    from pychem_gb300 import workloads as W
    if name.startswith("water"):
        n = {"water1": (1, 1, 1), "water2": (2, 1, 1), "water8": (2, 2, 2)}[name]
        return W.water_cluster(*n, seed=4)
    if name == "linear":      # integrals that vanish by symmetry
        return [["C", 6.0, 0.0, 0.0, 0.0], ["C", 6.0, 0.0, 0.0, 1.25]]
    return W.alkane(int(name[6:]), seed=4)


@pytest.mark.parametrize("name,basis,precision", [
    ("water1", "STO-3G", "fp64"), ("water2", "6-31G", "fp64"), ("linear", "cc-pVDZ", "fp64"), ("alkane3", "cc-pVDZ", "fp64"),
    ("alkane3", "6-31G", "mixed"), ("water8", "6-31G", "fp64"), ("water8", "6-31G", "mixed")])
def test_fock_matrices(name, basis, precision):
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    eng = GpuEngine(Molecule(_coords(name), basis), precision=precision).prepare()
    n = eng.nbf
    eri = eng.dense_eri().reshape(n * n, n, n)
    g = torch.Generator(device="cuda").manual_seed(n)
    D = torch.randn(2, n, n, dtype=torch.float64, device="cuda", generator=g)
    D = 0.25 * (D + D.transpose(1, 2))

    def J(d):
        return (eri.reshape(n * n, n * n) @ d.reshape(-1)).reshape(n, n)

    def K(d):
        return torch.einsum("abcd,bd->ac", eri.reshape(n, n, n, n), d)

    F = eng.fock(D[0])
    assert float((F - (eng.H + 2 * J(D[0]) - K(D[0]))).abs().max()) < 2e-11
    Fa, Fb = eng.fock_u(D[0], D[1])
    Jt = J(D[0] + D[1])
    assert float((Fa - (eng.H + Jt - K(D[0]))).abs().max()) < 2e-11
    assert float((Fb - (eng.H + Jt - K(D[1]))).abs().max()) < 2e-11


def test_scaling_at_the_ends_of_the_range():
    """Densities with zeros, tiny and infinite elements: what the products give."""
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    eng = GpuEngine(Molecule(_coords("water1"), "STO-3G")).prepare()
    n = eng.nbf
    assert torch.equal(eng.fock(torch.zeros(n, n, dtype=torch.float64, device="cuda")), eng.H)
    D = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    D[2, 2] = 1e-300
    assert float((eng.fock(D) - eng.H).abs().max()) < 1e-290 + 1e-15 * float(eng.H.abs().max())
    D[2, 2] = float("inf")
    F = eng.fock(D)
    assert not torch.isfinite(F[2, 2]) and bool(torch.isfinite(eng.H).all())
    D[2, 2] = float("nan")
    assert torch.isnan(eng.fock(D)[2, 2])
