"""Integral kernels with a quartet's primitives spread over several lanes, and the table
ranges of their fundamentals, against one lane per quartet and against the CPU oracle.

Tolerances: sums of at most 1,296 primitive terms of size 5 in another order differ by
less than 1296 * 2^-53 * 5 = 7e-13 (2e-12 asked); against the oracle 1e-12 for 1/r12
(its own error is 1e-13), and 1e-10 for j0(S r12), where the oracle keeps the 20-term
series of the reference (truncated at up to 2e-11 just below S r = 10).
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ANGSTROM = 1.8897161646320724


def _engine(coords, basis):
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    electrons = int(sum(a[1] for a in coords))
    eng = GpuEngine(Molecule(coords, basis, multiplicity=1 + electrons % 2))
    eng.one_electron()
    return eng


def _blocks(eng, cls, tasks, n, more, S):
    from pychem_gb300 import _lib
    from pychem_gb300.engine import _ptr, _stream
    store = torch.full((_lib.load().pcg_eri_class_nout(cls) * n,), float("nan"), dtype=torch.float64, device="cuda")
    b, p = ctypes.byref(eng.basis_t), ctypes.byref(eng.pairs_t)
    if S is None:
        _lib.call("pcg_eri_class_split", cls, b, p, _ptr(tasks), n, (ctypes.c_int * 6)(*more), _ptr(store), 0, _stream())
    else:
        eng.scattering = S
        fac = eng._scattering_factors()
        eng.scattering = None
        _lib.call("pcg_scattering_class_split", cls, b, p, _ptr(fac), _ptr(tasks), n, (ctypes.c_int * 6)(*more), S, _ptr(store), _stream())
    return store.view(-1, n)


@pytest.mark.parametrize("S", [None, 1.7])
@pytest.mark.parametrize("basis", ["6-31G", "cc-pVDZ"])
def test_lanes_of_a_quartet(basis, S):
    """Prefix lengths around warp and task boundaries, lists long enough for one lane a
    quartet and short ones, whole lists of one class."""
    from pychem_gb300 import workloads
    eng = _engine(workloads.water(), basis)
    eng.schwarz()
    eng.build_tasks()
    for cls, rec in eng.classes.items():
        tasks, n = rec["64"]
        many = tasks.view(n, 2).repeat(-(-45000 // n), 1).contiguous().view(-1)   # > 40,000: one lane each
        ref = _blocks(eng, cls, many, many.numel() // 2, (0,) * 6, S)[:, :n]
        scale = float(ref.abs().max())
        for k in sorted({1, min(2, n), min(33, n), n}):
            for more in sorted({tuple(min(k, x) for x in m) for m in ((0, 0, 0, 0, 0, 0), (1, 1, 1, 1, 1, 1), (0, 0, 0, 0, 0, 1),
                                (0, 0, k // 2, k, k, k), (k // 2, k // 2, k, k, k, k), (1, 2, 3, 4, 5, 6), (k, k, k, k, k, k))}):
                got = _blocks(eng, cls, tasks, k, more, S)
                assert float((got - ref[:, :k]).abs().max()) <= 2e-12 * max(1.0, scale), (cls, k, more)


@pytest.mark.parametrize("S", [None, 0.0, 0.5, 6.0, 40.0])
def test_fundamentals_over_distance(S):
    """Separations that put T on both sides of 48 and z = S r on both sides of 10 and 100,
    coincident centres and grid points included."""
    from oracle import oracle as O
    for r in (0.0009765625, 0.25, 0.5, 1.0, 1.625, 2.5, 2.51, 5.0, 6.9, 7.0, 11.0, 30.0):
        coords = [["H", 1.0, 0.1, -0.2, 0.3], ["O", 8.0, 0.1, -0.2 + 0.6 * r, 0.3 + 0.8 * r]]
        eng = _engine(coords, "6-31G")
        eng.scattering = S
        eng.threshold = 0.0
        eng.schwarz()
        eng.build_tasks()
        eng.compute_eris()
        eng.scattering = None
        got = eng.dense_eri().cpu().numpy()
        b = O.Basis([(a[0], a[1], *[v * ANGSTROM for v in a[2:]]) for a in coords], "6-31G")
        ref = b.eri_dense(scattering=S) if S is not None else b.eri_dense()
        keep = np.abs(got) > 0           # the oracle leaves out what its threshold screens
        assert np.abs((got - ref)[keep & (np.abs(ref) > 0)]).max() < (1e-12 if S is None else 1e-10), r


@pytest.mark.parametrize("most", [0, 20, 1024])
def test_exponent_sum_table(most, monkeypatch):
    """No table, a table that is refused for its size, and a whole one give the same blocks
    (each factor to a few roundings: 1e-14 of the largest integral)."""
    from pychem_gb300 import engine, workloads
    coords = workloads.water() + [["C", 6.0, 3.0, 0.0, 0.5], ["H", 1.0, 3.0, 1.0, 0.0], ["H", 1.0, 3.5, -0.5, 0.8]]
    ref = _engine(coords, "cc-pVDZ").prepare()
    monkeypatch.setattr(engine, "MAX_EXPONENT_SUMS", most)
    got = _engine(coords, "cc-pVDZ").prepare()
    assert (got.prim_t.nz > 0) == (most == 1024)
    for key, store in ref.stores.items():
        assert float((got.stores[key] - store).abs().max()) < 1e-14 * max(1.0, float(store.abs().max())) * 30
    # sums that the table lacks are computed
    part = got.pd["zid"].clone()
    part[::3] = -1
    got.pd["zid"] = part
    got.prim_t.zid = part.data_ptr()
    got.compute_eris()
    for key, store in ref.stores.items():
        assert float((got.stores[key] - store).abs().max()) < 1e-14 * max(1.0, float(store.abs().max())) * 30
