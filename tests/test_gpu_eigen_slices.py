"""Single matrices of 65 to 136 rows whose spectra leave little to slice at: levels a few 1e-6
to 1e-3 of the largest apart, two clusters, and levels graded over 12 decades.

Tolerance: residuals 1e-12 of the norm and orthogonality 1e-13, the bars of test_gpu_eigen.py."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def spectra(n):
    for gap in (1e-3, 1e-4, 3e-5, 1.2e-5, 5e-6):
        yield 1.0 + gap * np.arange(n)
    yield 10.0 ** np.linspace(-12.0, 0.0, n)
    yield np.concatenate([np.zeros(n // 2), np.full(n - n // 2, 2.1e-5)]) + 1.0


@pytest.mark.parametrize("n", [65, 104, 136])
def test_exact_whatever_the_gaps(n):
    from pychem_gb300 import eigen
    Q = torch.tensor(np.linalg.qr(np.random.default_rng(n).standard_normal((n, n)))[0], device="cuda")
    for lam in spectra(n):
        lam = torch.tensor(lam, device="cuda")
        A = (Q * lam) @ Q.T
        A = 0.5 * (A + A.T)
        for X in (None, Q):
            w, V = eigen.eigh(A, X_prev=X)
            size = float(lam.abs().max())
            assert float((w - lam).abs().max()) < 1e-12 * size
            assert float((A @ V - V * w).abs().max()) < 1e-12 * size
            assert float((V.T @ V - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max()) < 1e-13


@pytest.mark.parametrize("n", [33, 64, 65, 80, 81])
def test_slicing_itself(n):
    """Below the size from which single matrices are sliced by themselves, too."""
    from pychem_gb300 import eigen
    Q = torch.tensor(np.linalg.qr(np.random.default_rng(n).standard_normal((n, n)))[0], device="cuda")
    for lam in spectra(n):
        lam = torch.tensor(lam, device="cuda")
        A = (Q * lam) @ Q.T
        A = 0.5 * (A + A.T)
        for w, V in (eigen.exact_eigh(A), eigen.eigh(A)):
            size = float(lam.abs().max())
            assert float((w - lam).abs().max()) < 1e-12 * size
            assert float((A @ V - V * w).abs().max()) < 1e-12 * size
            assert float((V.T @ V - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max()) < 1e-13
