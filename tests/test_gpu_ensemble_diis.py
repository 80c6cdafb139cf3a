"""Ensemble SCF over the DIIS depths that the caller may ask for, none among them: the same energies
(1e-8, a hundred times the stop test's)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_depths():
    from pychem_gb300.ensemble import EnsembleEngine, rhf_batched
    from pychem_gb300.molecule import Molecule
    mols = [Molecule([["H", 1.0, 0.0, 0.0, 0.0], ["H", 1.0, 0.0, 0.0, 0.7 + 0.05 * k]], "6-31G") for k in range(5)]
    want = None
    for depth in (8, 0, 1, 2, 32, 40):
        r = rhf_batched(EnsembleEngine(mols).prepare(), diis_size=depth)
        assert r.converged.all()
        want = r.E if want is None else want
        assert np.abs(r.E - want).max() < 1e-8
