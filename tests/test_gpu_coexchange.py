"""J and K of co-densities by products with pair matrices, at and around the numbers of
densities and functions where the route changes, against the dense contractions and against the
digestion; the tiled matrix product at the edges of its tiles.

Tolerance: sums of up to n^2 products of |W| < 5 with integrals of total magnitude below 1e3:
2^-53 * n * 5e3 = 2.4e-11 at n = 43 (5e-11 asked)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd", [1, 2, 15, 16, 17, 64, 129])
@pytest.mark.parametrize("name,basis", [("h2", "STO-3G"), ("water", "6-31G"), ("c2", "cc-pVDZ"), ("alkane", "6-31G")])
def test_coulomb_exchange(name, basis, nd, monkeypatch):
    from pychem_gb300 import engine, workloads
    from pychem_gb300.molecule import Molecule
    coords = {"h2": [["H", 1.0, 0, 0, 0], ["H", 1.0, 0, 0, 0.74]], "water": workloads.water(),
              "c2": [["C", 6.0, 0, 0, 0], ["C", 6.0, 0, 0, 1.25]], "alkane": workloads.alkane(3)}[name]
    eng = engine.GpuEngine(Molecule(coords, basis)).prepare()
    n = eng.nbf
    g = torch.Generator(device="cuda").manual_seed(nd)
    W = torch.randn(nd, n, n, dtype=torch.float64, device="cuda", generator=g)
    eri = eng.dense_eri()
    Jr = (W.reshape(nd, n * n) @ eri.reshape(n * n, n * n)).reshape(nd, n, n)
    Kr = torch.einsum("abcd,xcb->xad", eri, W)
    for least in (engine.COEXCHANGE_MIN, 10 ** 9, 1):
        monkeypatch.setattr(engine, "COEXCHANGE_MIN", least)
        for w in (W, W.transpose(1, 2).contiguous().transpose(1, 2)):
            J, K = eng.coulomb_exchange(w)
            assert J.shape == K.shape == W.shape
            assert float((J - Jr).abs().max()) < 5e-11 and float((K - Kr).abs().max()) < 5e-11


@pytest.mark.parametrize("M,N,K", [(32, 32, 1), (64, 64, 64), (65, 95, 65), (97, 128, 79), (756, 406, 406), (63, 64, 64)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_tiled_product(M, N, K, ta, tb):
    """Batches large enough for the 32 x 32 tiles; sums of K products of normal deviates:
    K 2^-53 * 16 < 1e-12."""
    from pychem_gb300.dense import mm
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    batch = 100 if M < 200 else 3
    A = torch.randn(batch, *((K, M) if ta else (M, K)), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn(batch, *((N, K) if tb else (K, N)), dtype=torch.float64, device="cuda", generator=g)
    out = torch.randn(batch, N, M, dtype=torch.float64, device="cuda", generator=g).transpose(1, 2)
    ref = (A.transpose(1, 2) if ta else A) @ (B.transpose(1, 2) if tb else B)
    want = 2.0 * ref - 0.5 * out
    assert float((mm(A, B, ta=ta, tb=tb) - ref).abs().max()) < 1e-12 * max(1, K)
    assert float((mm(A, B, ta=ta, tb=tb, out=out, alpha=2.0, beta=-0.5) - want).abs().max()) < 1e-12 * max(1, K)
