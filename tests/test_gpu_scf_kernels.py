"""The dense kernels of an SCF iteration at the edges of their tiles and blocks, and the Jacobi
solver over scales, clusters and the CTAs that share a matrix.

Tolerances: products as sums of K terms (1e-13 K max|a| max|b|); eigenvalues and residuals
1e-12 of the norm and orthogonality 1e-13, the bars of test_gpu_eigen.py."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
F64 = dict(dtype=torch.float64, device="cuda")


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("M,K", [(1, 1), (7, 3), (8, 32), (9, 33), (64, 80), (137, 137), (208, 80)])
@pytest.mark.parametrize("ta", [False, True])
def test_symmetric_product(M, K, ta):
    from pychem_gb300.dense import mm
    A = torch.randn(*((K, M) if ta else (M, K)), generator=_gen(M), **F64)
    out = torch.randn(M, M, generator=_gen(K), **F64)
    out = out + out.T
    ref = A.T @ A if ta else A @ A.T
    kw = dict(ta=True) if ta else dict(tb=True)
    got = mm(A, A, sym=True, **kw)
    assert torch.equal(got, got.T)
    tol = 1e-13 * K * float(A.abs().max()) ** 2
    assert float((got - ref).abs().max()) <= tol
    want = 2.0 * ref - 0.5 * out
    got = mm(A, A, sym=True, out=out, alpha=2.0, beta=-0.5, **kw)
    assert float((got - want).abs().max()) <= 4 * tol + 1e-14


@pytest.mark.parametrize("n,n2", [(1, 1), (13, 13), (15, 12), (16, 16), (17, 17), (128, 128), (208, 205)])
@pytest.mark.parametrize("nan", [False, True])
def test_scf_stats(n, n2, nan):
    from pychem_gb300 import _lib
    from pychem_gb300._stream import stream
    g = _gen(n)
    D, H, F, Dold = (torch.randn(n, n, generator=g, **F64) for _ in range(4))
    P = torch.randn(n2, n2, generator=g, **F64)
    if nan:
        P[n2 // 2, 0] = float("nan")
    R, part, vals = torch.empty(n2, n2, **F64), torch.empty(192, **F64), torch.full((6,), 7.0, **F64)
    want = (torch.sum(D * (H + F)), torch.sqrt(torch.mean((D - Dold) ** 2)), (P - P.T).abs().amax())
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.call("pcg_scf_stats", n, n2, p(P), p(D), p(H), p(F), p(Dold), p(R), p(part), p(vals), stream())
    assert torch.equal(R.nan_to_num(9.0), (P - P.T).nan_to_num(9.0)) and torch.equal(Dold, D)
    assert abs(float(vals[0] - want[0])) < 1e-11 * n and abs(float(vals[1] - want[1])) < 1e-12
    assert bool(torch.isnan(vals[5])) == nan and (nan or float(vals[5]) == float(want[2]))
    assert vals[2:5].tolist() == [7.0, 7.0, 7.0]


@pytest.mark.parametrize("n,nocc", [(2, 1), (31, 7), (33, 32), (208, 80)])
def test_projector_check(n, nocc):
    from pychem_gb300.dense import projector_check
    S, R = (torch.randn(n, n, generator=_gen(n + k), **F64) for k in (0, 1))
    d = torch.diagonal(S)
    want = torch.stack([R.abs().amax(), S[:nocc, nocc:].abs().amax(), d[:nocc].amax() - d[nocc:].amin()])
    assert torch.equal(projector_check(S, R, nocc), want)
    S[0, n - 1] = float("nan")
    assert bool(torch.isnan(projector_check(S, R, nocc)).all())


@pytest.mark.parametrize("n,batch", [(2, 1), (13, 1), (30, 1), (30, 200), (64, 3), (104, 1), (136, 1), (136, 160)])
@pytest.mark.parametrize("scale", [1.0, 1e-150, 1e150])
def test_fp64_jacobi(n, batch, scale):
    from pychem_gb300 import eigen
    M = torch.randn(batch, n, n, generator=_gen(n + batch), **F64)
    A = M + M.transpose(1, 2)
    A[0].fill_(1.0)                                   # equal diagonal elements, one large cluster
    if batch > 1:
        A[1] = torch.diag(torch.arange(n, **F64))     # nothing to rotate
    if batch > 2:                                     # near-degenerate and far-off levels
        A[2] = 1e-9 * A[2] + torch.diag(torch.cat([torch.full((n // 2,), -20.0, **F64), torch.full((n - n // 2,), 1e3, **F64)]))
    w, V = eigen.eigh(A * scale)
    w = w / scale
    ref = torch.linalg.eigvalsh(A)
    size = ref.abs().amax(dim=1, keepdim=True).clamp_min(1e-30)
    assert float(((w - ref).abs() / size).max()) < 1e-12
    assert float(((A @ V - V * w.unsqueeze(1)).abs() / size.unsqueeze(2)).max()) < 1e-12
    assert float((V.transpose(1, 2) @ V - torch.eye(n, **F64)).abs().max()) < 1e-13


@pytest.mark.parametrize("n,batch", [(8, 1), (100, 1), (208, 1), (208, 5), (298, 1), (334, 2)])
def test_fp32_jacobi_shared_matrix(n, batch):
    from pychem_gb300 import eigen
    M = torch.randn(batch, n, n, generator=_gen(n), **F64)
    A = M + M.transpose(1, 2)
    w, V = eigen.jacobi(A, fp32=True)
    size = float(A.abs().amax()) * n ** 0.5
    assert float((V.transpose(1, 2) @ V - torch.eye(n, **F64)).abs().max()) < 1e-4
    assert float((A @ V - V * w.unsqueeze(1)).abs().max()) < 1e-4 * size


@pytest.mark.parametrize("n", [32, 33, 52, 64, 65, 104, 136])
@pytest.mark.parametrize("scale", [1.0, 1e-150, 1e150])
def test_one_matrix(n, scale):
    """Both sides of the sizes where a single matrix changes route; a cluster of equal levels."""
    from pychem_gb300 import eigen
    Q, _ = torch.linalg.qr(torch.randn(n, n, generator=_gen(n), **F64))
    lam = torch.linspace(-2.0, 5.0, n, **F64)
    lam[: n // 4] = -20.0
    A = (Q * lam) @ Q.T
    A = 0.5 * (A + A.T)
    for X in (None, Q):
        w, V = eigen.eigh(A * scale, X_prev=X)
        w = w / scale
        assert float((w - lam).abs().max()) < 2e-11
        assert float((A @ V - V * w).abs().max()) < 2e-11
        assert float((V.T @ V - torch.eye(n, **F64)).abs().max()) < 1e-13
    w, V = eigen.eigh(torch.zeros(n, n, **F64))
    assert float(w.abs().max()) == 0.0 and float((V.T @ V - torch.eye(n, **F64)).abs().max()) < 1e-13


@pytest.mark.parametrize("atoms", [6, 8])
def test_rhf_without_virtual_orbitals(atoms):
    """Every orbital occupied (neon atoms in a minimal basis, 30 and 40 functions)."""
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    from pychem_gb300.scf import rhf
    one = rhf(GpuEngine(Molecule([["NE", 10.0, 0.0, 0.0, 0.0]], "STO-3G")).prepare()).E
    r = rhf(GpuEngine(Molecule([["NE", 10.0, 30.0 * k, 0.0, 0.0] for k in range(atoms)], "STO-3G")).prepare())
    assert r.converged and abs(r.E - atoms * one) < 1e-7


@pytest.mark.parametrize("n", [40, 65, 100, 136])
def test_one_matrix_without_gaps(n):
    """Multiples of the identity, and clusters wider than a part of the sliced spectrum."""
    from pychem_gb300 import eigen
    Q, _ = torch.linalg.qr(torch.randn(n, n, generator=_gen(n), **F64))
    for lam in (torch.ones(n, **F64), torch.cat([torch.zeros(n - 3, **F64), torch.ones(3, **F64)]),
                1.0 + 1e-9 * torch.arange(n, **F64)):
        A = (Q * lam) @ Q.T
        A = 0.5 * (A + A.T)
        w, V = eigen.eigh(A)
        assert float((w - lam).abs().max()) < 1e-12
        assert float((A @ V - V * w).abs().max()) < 1e-12
        assert float((V.T @ V - torch.eye(n, **F64)).abs().max()) < 1e-13


def test_rhf_without_a_gap():
    """A square of hydrogen atoms (degenerate frontier orbitals) among distant helium atoms, 36
    functions: the route with refined vectors gives the Jacobi route's energies."""
    from pychem_gb300 import eigen
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    from pychem_gb300.scf import rhf
    coords = [["H", 1.0, x, y, 0.0] for x in (0.0, 1.2) for y in (0.0, 1.2)]
    coords += [["HE", 2.0, 6.0 + 3.0 * k, 0.0, 0.0] for k in range(14)]
    eng = GpuEngine(Molecule(coords, "6-31G")).prepare()
    assert eng.nbf > eigen.FP64_JACOBI_ONE_N
    got = rhf(eng, max_iter=60)
    old = eigen.FP64_JACOBI_ONE_N
    eigen.FP64_JACOBI_ONE_N = eigen.FP64_JACOBI_MAX_N
    try:
        want = rhf(eng, max_iter=60)
    finally:
        eigen.FP64_JACOBI_ONE_N = old
    assert bool(torch.isfinite(got.eps).all()) and bool(torch.isfinite(got.D).all())
    assert got.converged == want.converged
    assert not want.converged or abs(got.E - want.E) < 1e-7


@pytest.mark.parametrize("batch,mo,mn", [(1, 0, 1), (3, 1, 2), (5, 7, 8), (6, 8, 8), (130, 8, 8), (2, 31, 32), (2, 32, 32)])
def test_diis_batched(batch, mo, mn):
    """Coefficients and the moved matrix against the host's solve: 64 eps times the condition
    of the scaled system."""
    from pychem_gb300 import _lib
    from pychem_gb300.engine import _ptr
    from pychem_gb300._stream import stream
    from pychem_gb300.scf import diis_coefficients_batched
    rng = np.random.default_rng(mo)
    r = rng.standard_normal((batch, mo + 1, 3 * mo + 4)) * 0.5 ** np.arange(mo + 1)[:, None]
    G = np.einsum("bik,bjk->bij", r, r)
    old = torch.tensor(G[:, :mo, :mo].copy(), device="cuda")
    row = torch.zeros(batch, mo + 3, dtype=torch.float64, device="cuda")
    row[:, 2:] = torch.tensor(G[:, mo, :].copy())
    new = torch.empty(batch, mn, mn, dtype=torch.float64, device="cuda")
    coef = torch.empty(batch, mn, dtype=torch.float64, device="cuda")
    _lib.call("pcg_diis_batched", batch, mo, mn, _ptr(old), _ptr(row[:, 2:]), row.stride(0), _ptr(new), _ptr(coef), stream())
    cut = mo + 1 - mn
    assert np.array_equal(new.cpu().numpy(), G[:, cut:, cut:])
    want = diis_coefficients_batched(G[:, cut:, cut:])
    M = -np.ones((batch, mn + 1, mn + 1))
    M[:, :mn, :mn] = G[:, cut:, cut:] / np.abs(np.diagonal(G[:, cut:, cut:], axis1=1, axis2=2)).max(1)[:, None, None]
    M[:, mn, mn] = 0.0
    tol = 64 * 2.2e-16 * np.linalg.cond(M)
    assert (np.abs(coef.cpu().numpy() - want).max(1) <= tol * np.maximum(1.0, np.abs(want).max(1))).all()


def test_diis_batched_drops_repeats():
    """Residuals that repeat exactly: the newest alone is used."""
    from pychem_gb300 import _lib
    from pychem_gb300.engine import _ptr
    from pychem_gb300._stream import stream
    G = np.ones((2, 3, 3))
    G[1] = 0.0
    old = torch.tensor(G[:, :2, :2].copy(), device="cuda")
    row = torch.tensor(G[:, 2, :].copy(), device="cuda")
    new = torch.empty(2, 3, 3, dtype=torch.float64, device="cuda")
    coef = torch.empty(2, 3, dtype=torch.float64, device="cuda")
    _lib.call("pcg_diis_batched", 2, 2, 3, _ptr(old), _ptr(row), 3, _ptr(new), _ptr(coef), stream())
    assert coef.cpu().tolist() == [[0.0, 0.0, 1.0]] * 2
