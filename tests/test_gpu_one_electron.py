"""Primitive-pair data and one-electron matrices of the per-class kernels.

Tolerances: zeta and 1/(2 zeta) are one operation each; K is 1e-13 times the size of the
exponent's argument (a rounding of the argument is one of the result), argument below 700;
matrix elements are sums of at most 81 primitive terms and 40 nuclei, 1e-12 of the largest."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _engine(coords, basis):
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    electrons = int(sum(a[1] for a in coords))
    return GpuEngine(Molecule(coords, basis, multiplicity=1 + electrons % 2))


def _water():
    from pychem_gb300 import workloads
    return workloads.water()


@pytest.mark.parametrize("copies,basis", [(1, "6-31G"), (1, "cc-pVDZ"), (14, "cc-pVDZ"), (45, "6-31G")])
def test_pair_data(copies, basis):
    """1 to 32 shell pairs to a warp."""
    coords = [[*a[:4], a[4] + 5.0 * k] for k in range(copies) for a in _water()]
    eng = _engine(coords, basis)
    a, h, f = eng.h_basis, eng.h_pairs, eng.pd_full
    p = np.repeat(np.arange(len(h["A"])), h["npp"])
    loc = np.arange(len(p)) - h["ppoff"][p]
    A, B = h["A"][p], h["B"][p]
    nb = a["sh_nprim"][B]
    ia, ib = a["sh_prim"][A] + loc // nb, a["sh_prim"][B] + loc % nb
    al, be = a["pr_exp"][ia], a["pr_exp"][ib]
    xyz = a["sh_xyz"].reshape(-1, 3)
    z = al + be
    arg = al * be / z * ((xyz[A] - xyz[B]) ** 2).sum(1)
    K = a["pr_cc"][ia] * a["pr_cc"][ib] * np.sqrt(2 / np.sqrt(np.pi)) * (np.pi / z) ** 1.5 * np.exp(-arg) * np.sqrt(z)
    P = (al[:, None] * xyz[A] + be[:, None] * xyz[B]) / z[:, None]
    assert np.array_equal(f["zeta"].cpu().numpy(), z)
    assert np.allclose(f["oo2z"].cpu().numpy(), 0.5 / z, rtol=1e-15, atol=0)
    assert np.abs(f["P"].cpu().numpy().reshape(-1, 3) - P).max() <= 1e-13 * max(1.0, np.abs(xyz).max())
    near = arg < 700
    assert (np.abs(f["K"].cpu().numpy() - K)[near] <= (1e-13 * (1 + arg) * np.abs(K))[near]).all()


@pytest.mark.parametrize("basis", ["6-31G", "cc-pVDZ"])
def test_one_electron_pair_order(basis):
    """The shells of a pair in either order, and every pair launched alone."""
    from pychem_gb300 import _lib
    from pychem_gb300.engine import _ptr, _stream
    eng = _engine(_water(), basis)
    S0, H0 = eng.one_electron()
    n = S0.shape[-1]
    A, B = eng.pd["A"], eng.pd["B"]

    def run(x, y):
        S, H = (torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(2))
        for lo in range(0, len(x)):
            _lib.call("pcg_one_electron", ctypes.byref(eng.basis_t), 1, _ptr(x[lo:]), _ptr(y[lo:]), _ptr(S), _ptr(H), _stream())
        return S, H

    S1, H1 = run(A, B)
    assert torch.equal(S1, S0) and torch.equal(H1, H0)
    S2, H2 = run(B, A)
    assert float((S2 - S0).abs().max()) <= 1e-12
    assert float((H2 - H0).abs().max()) <= 1e-12 * float(H0.abs().max())
    assert torch.equal(S2, S2.T) and torch.equal(H2, H2.T)


@pytest.mark.parametrize("npair", [1, 2, 31, 1025, 40000])
def test_pair_flags(npair):
    """Against the definition, exactly: one pair (no other), repeated and zero factors."""
    from pychem_gb300 import _lib
    from pychem_gb300.engine import _ptr, _stream
    rng = np.random.default_rng(npair)
    for kind in range(3):
        Q = rng.random(npair) ** 8
        if kind == 1:
            Q[rng.integers(npair, size=2)] = 2.0
        if kind == 2:
            Q[:] = np.where(rng.random(npair) < 0.5, 0.0, 1.0)
        sp = rng.integers(npair, size=2 * npair + 3)
        best = np.argmax(Q)
        rest = np.delete(Q, best)
        for thr in (0.0, 0.1, -1.0):
            want = np.zeros(npair, dtype=bool) if npair == 1 else Q * np.where(np.arange(npair) == best, rest.max(), Q[best]) > thr
            flag = torch.full((len(sp),), -7, dtype=torch.int32, device="cuda")
            Qd, spd = torch.tensor(Q, device="cuda"), torch.tensor(sp, device="cuda")
            _lib.call("pcg_pair_flags", npair, _ptr(Qd), thr, len(sp), _ptr(spd), _ptr(flag), _stream())
            assert np.array_equal(flag.cpu().numpy(), want[sp].astype(np.int32)), (kind, thr)
