"""FP64 products of more rows than a grid has rows of tiles.  Tolerance: K 2^-53 of the sums of
magnitudes, twice."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(524281, 3, 5), (600001, 70, 65)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
def test_tall_product(M, N, K, ta, tb):
    from pychem_gb300.dense import mm
    g = torch.Generator(device="cuda").manual_seed(N)
    A = torch.randn(*((K, M) if ta else (M, K)), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn(*((N, K) if tb else (K, N)), dtype=torch.float64, device="cuda", generator=g)
    a, b = A.T if ta else A, B.T if tb else B
    out = torch.randn(M, N, dtype=torch.float64, device="cuda", generator=g)
    want = 2.0 * (a @ b) - 0.5 * out
    tol = 2.0 * K * 2.0 ** -53 * (2.0 * (a.abs() @ b.abs()) + out.abs())
    assert bool(((mm(A, B, ta=ta, tb=tb, out=out, alpha=2.0, beta=-0.5) - want).abs() <= tol).all())
