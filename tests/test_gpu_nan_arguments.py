"""NaN coordinates of either sign stay NaNs: the Boys and Bessel tables are not indexed by them."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NANS = [float("nan"), float(np.copysign(np.nan, -1.0))]


@pytest.mark.parametrize("nan", NANS, ids=["+", "-"])
@pytest.mark.parametrize("m", range(9))
def test_boys_orders(nan, m):
    from pychem_gb300 import _lib
    n = 70
    P = np.zeros((n, 3))
    P[:, 0] = np.linspace(0.5, 12.0, n)
    want = np.zeros((m + 1, n))
    got = np.zeros((m + 1, n))
    one, U, R, q = np.ones(n), np.ones(n), np.zeros((n, 3)), np.zeros((1, 3))
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    for out in (want, got):
        if out is got:
            P[::3, 1] = nan
        assert _lib.load().pcg_two_electron_fundamentals(p(out), p(one), p(U), p(P), p(one), p(U), p(q), p(R), n, 1, 1, 1,
                                                         m, 0, 0.0) == 0
    bad = np.zeros(n, dtype=bool)
    bad[::3] = True
    assert np.isnan(got[:, bad]).all() and np.array_equal(got[:, ~bad], want[:, ~bad])


@pytest.mark.parametrize("nan", NANS, ids=["+", "-"])
@pytest.mark.parametrize("basis", ["STO-3G", "cc-pVDZ"])
def test_one_electron(nan, basis):
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    coords = [["H", 1.0, 0.0, 0.0, 0.0], ["H", 1.0, 0.0, 0.0, 0.74], ["HE", 2.0, 1.5, nan, 0.0]]
    S, H = GpuEngine(Molecule(coords, basis)).one_electron()
    n = GpuEngine(Molecule(coords[:2], basis)).nbf
    assert bool(torch.isfinite(S[:n, :n]).all()) and bool(torch.isnan(H[:n, :n]).all())
    assert bool(torch.isnan(S[:n, n:]).any())


@pytest.mark.parametrize("nan", NANS, ids=["+", "-"])
@pytest.mark.parametrize("basis", ["STO-3G", "cc-pVDZ"])
def test_engine_without_primitive_pairs(nan, basis):
    """The largest primitive-pair factor is then a NaN and no pair is kept: integrals are zeros,
    Fock matrices NaNs."""
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    coords = [["HE", 2.0, 0.0, 0.0, 0.0], ["HE", 2.0, 1.5, nan, 0.0]]
    for precision in ("fp64", "mixed"):
        eng = GpuEngine(Molecule(coords, basis), precision=precision).prepare()
        assert eng.pd["zeta"].numel() == 0 and float(eng.Q.abs().max()) == 0.0
        assert bool(torch.isnan(eng.fock(torch.eye(eng.nbf, dtype=torch.float64, device="cuda"))).all())
    eng.scattering = 1.3
    assert float(eng.schwarz().abs().max()) == 0.0
