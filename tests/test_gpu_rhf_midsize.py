"""RHF of 33 to 136 functions, whose orbitals are refined from FP32 vectors: densities and
orbital energies of the route that solves every iteration by the FP64 Jacobi kernel.

Tolerance: an iteration's coupling between the spaces is at most 1e-12 of the largest Fock
element (20), over gaps of 0.4: 5e-11 an element of the density, and the stop test passes in the same
iteration; 5e-10 of the norm."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [("water", 3, "6-31G", 39), ("water", 4, "6-31G", 52), ("alkane", 5, "6-31G", 69), ("alkane", 3, "cc-pVDZ", 82),
         ("water", 8, "6-31G", 104), ("water", 16, "STO-3G", 112), ("alkane", 10, "6-31G", 134)]


@pytest.mark.parametrize("system,units,basis,n", CASES)
@pytest.mark.parametrize("graph", [None, False])
def test_same_as_jacobi_route(system, units, basis, n, graph):
    from pychem_gb300 import eigen, workloads
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    from pychem_gb300.scf import rhf
    if system == "water":
        nx, ny, nz = {3: (3, 1, 1), 4: (2, 2, 1), 8: (2, 2, 2), 16: (4, 2, 2)}[units]
        coords = workloads.water_cluster(nx=nx, ny=ny, nz=nz, seed=3)
    else:
        coords = workloads.alkane(units, seed=3)
    eng = GpuEngine(Molecule(coords, basis)).prepare()
    assert eng.nbf == n
    got = rhf(eng, graph=graph)
    old = eigen.FP64_JACOBI_ONE_N
    eigen.FP64_JACOBI_ONE_N = eigen.FP64_JACOBI_MAX_N
    try:
        want = rhf(eng, graph=graph)
    finally:
        eigen.FP64_JACOBI_ONE_N = old
    assert got.converged and want.converged and got.iterations == want.iterations
    for key in ("D", "eps"):
        a, b = got[key], want[key]
        assert float((a - b).norm() / b.norm()) < 5e-10


@pytest.mark.parametrize("gap", [True, False])
def test_refined_below_its_sizes(gap, monkeypatch):
    """36 functions with refined vectors, which go to the FP64 kernel by themselves: helium atoms, and
    with a square of hydrogen atoms whose frontier orbitals are degenerate."""
    from pychem_gb300 import eigen
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    from pychem_gb300.scf import rhf
    coords = [["H", 1.0, x, y if gap else 1.2 * (y > 0), 0.0] for x in (0.0, 1.2) for y in (0.0, 0.8)]
    coords += [["HE", 2.0, 6.0 + 3.0 * k, 0.0, 0.0] for k in range(14)]
    eng = GpuEngine(Molecule(coords, "6-31G")).prepare()
    want = rhf(eng, max_iter=60)
    monkeypatch.setattr(eigen, "REFINED_MIN_N", 0)
    got = rhf(eng, max_iter=60)
    assert eng.nbf == 36 and got.converged == want.converged
    assert bool(torch.isfinite(got.eps).all()) and bool(torch.isfinite(got.D).all())
    if gap:
        assert want.converged and got.iterations == want.iterations
        assert float((got.D - want.D).norm() / want.D.norm()) < 5e-10
    elif want.converged:
        assert abs(got.E - want.E) < 1e-7
