"""The network's tensor-core GEMM and weight gradient at the edges of their tiles, for every
operand layout the network uses, against 64-bit products.

Tolerance: each FP32 partial sum takes K/16 + 2 roundings of at most 2^-23 of the sum of
magnitudes, 2.2e-6 of sum |a||b| at K = 256 (4e-6 asked); the row sums of the weight gradient
add one rounding per partial (at most 38), 1e-5 asked.
"""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _call(name, *args):
    from pychem_gb300 import _lib
    return _lib.call(name, *[ctypes.c_void_p(a.data_ptr()) if torch.is_tensor(a) else a for a in args],
                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


def _rand(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g)


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 47, 31), (128, 64, 32), (129, 65, 33), (300, 256, 40),
                                   (515, 47, 256), (64, 256, 256), (257, 40, 47), (130, 96, 103)])
@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("bf16", [True, False])
def test_gemm(M, N, K, layout, bf16):
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 31 * K)
    A = _rand(g, K, M) if layout == "tn" else _rand(g, M, K)
    B = _rand(g, N, K) if layout == "nt" else _rand(g, K, N)
    A = A * torch.exp2(torch.randint(-12, 12, A.shape, device="cuda", generator=g).float())
    B = B.to(torch.bfloat16) if bf16 else B
    bias = _rand(g, N)
    Am, Bm = (A.T if layout == "tn" else A).double(), (B.T if layout == "nt" else B).double()
    ref, size = Am @ Bm, Am.abs() @ Bm.abs()
    sa = (1, M) if layout == "tn" else (K, 1)
    sb = (1, K) if layout == "nt" else (N, 1)
    nan = float("nan")

    def run(act=0, acc=0, b=None, Z=None, C=None):
        C = torch.full((M, N), nan, device="cuda") if C is None else C
        _call("pcg_mlp_gemm", M, N, K, A, *sa, B, int(bf16), *sb, C, N, acc, b, Z, act)
        return C.double()

    assert ((run() - ref).abs() <= 4e-6 * size).all()
    C0 = _rand(g, M, N)
    assert ((run(acc=1, C=C0.clone()) - (ref + C0.double())).abs() <= 4e-6 * (size + C0.abs())).all()
    Z = torch.full((M, N), nan, device="cuda")
    out = run(act=1, b=bias, Z=Z)
    z = ref + bias.double()
    assert ((Z.double() - z).abs() <= 4e-6 * (size + bias.abs())).all()
    assert ((out - z * torch.sigmoid(z)).abs() <= 6e-6 * (size + bias.abs() + 1)).all()
    Zin = _rand(g, M, N)
    s = torch.sigmoid(Zin.double())
    slope = s * (1 + Zin.double() * (1 - s))
    assert ((run(act=2, Z=Zin) - ref * slope).abs() <= 6e-6 * (size + 1e-6)).all()
    assert _status() == 0


def _status():
    from pychem_gb300 import _lib
    return _lib.load().pcg_mlp_status(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("M,K,N", [(1, 40, 256), (31, 256, 47), (128, 128, 64), (129, 129, 65), (4097, 256, 256),
                                   (10989, 40, 256), (5000, 1, 1)])
def test_weight_gradient(M, K, N):
    from pychem_gb300 import _lib
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    A, G = _rand(g, M, K), _rand(g, M, N)
    dW, db = torch.full((K, N), float("nan"), device="cuda"), torch.full((N,), float("nan"), device="cuda")
    ws = torch.empty(_lib.load().pcg_mlp_wgrad_workspace(M, K, N), dtype=torch.uint8, device="cuda")
    _call("pcg_mlp_wgrad", M, K, N, A, G, dW, db, ws, ws.numel())
    size = A.double().abs().T @ G.double().abs()
    assert ((dW.double() - A.double().T @ G.double()).abs() <= 1e-5 * size).all()
    assert ((db.double() - G.double().sum(0)).abs() <= 1e-5 * G.double().abs().sum(0)).all()


def test_infinities_and_nans():
    """A row with an infinity or a NaN gives what FP32 products give, and no other row."""
    g = torch.Generator(device="cuda").manual_seed(3)
    M, N, K = 130, 64, 40
    A, B = _rand(g, M, K), (_rand(g, K, N).abs() + 0.5).to(torch.bfloat16)
    A[1, 3], A[5, 39], A[129, 0], A[7, 2] = float("inf"), float("-inf"), float("nan"), 3.0e38
    A[9, 4] = torch.tensor([0x7F800001], dtype=torch.int32).view(torch.float32).item()
    C = torch.empty(M, N, device="cuda")
    _call("pcg_mlp_gemm", M, N, K, A, K, 1, B, 1, N, 1, C, N, 0, None, None, 0)
    ref = A @ B.float()
    assert torch.equal(torch.isnan(C), torch.isnan(ref))
    assert torch.equal(C[torch.isinf(ref)], ref[torch.isinf(ref)])


@pytest.mark.parametrize("N,K", [(256, 40), (250, 47)])
@pytest.mark.parametrize("layout", ["nn", "nt"])
@pytest.mark.parametrize("bf16", [True, False])
def test_gemm_wide_tiles(N, K, layout, bf16):
    """Tiles of 128 columns (more than 152 of 64), with rows and columns past the last tile."""
    test_gemm(5001, N, K, layout, bf16)


@pytest.mark.parametrize("M", [130, 5001])
@pytest.mark.parametrize("bf16", [True, False])
def test_infinite_weights(M, bf16):
    """Infinities in the other operand, against activations that are exact in one and in two BF16
    terms: infinities and NaNs where FP32 products have them."""
    from pychem_gb300 import _lib
    g = torch.Generator(device="cuda").manual_seed(M)
    N, K = 200, 40
    A = torch.randint(1, 9, (M, K), device="cuda", generator=g).float()
    A[::3] = A[::3] + 1.0 / 1024
    A[5, 7], A[6, 2] = 0.0, -1.5                       # 0 times an infinity is a NaN
    B = (_rand(g, K, N).abs() + 0.5)
    B[3, 11], B[39, 199], B[7, 64], B[2, 5] = float("inf"), float("-inf"), float("inf"), float("nan")
    B[0, 20], B[1, 20] = float("inf"), float("-inf")
    B = B.to(torch.bfloat16) if bf16 else B
    ref = A @ B.float()
    C = torch.empty(M, N, device="cuda")
    _call("pcg_mlp_gemm", M, N, K, A, K, 1, B, int(bf16), N, 1, C, N, 0, None, None, 0)
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isnan(C), torch.isnan(ref)) and torch.equal(C[torch.isinf(ref)], ref[torch.isinf(ref)])
    assert ((C - ref)[fin].abs() <= 4e-6 * (A.abs() @ B.float().abs())[fin]).all()
    G = _rand(g, M, N).abs()
    G[1, 3], G[M - 1, 199] = float("inf"), float("-inf")
    dW, db = torch.empty(K, N, device="cuda"), torch.empty(N, device="cuda")
    ws = torch.empty(_lib.load().pcg_mlp_wgrad_workspace(M, K, N), dtype=torch.uint8, device="cuda")
    _call("pcg_mlp_wgrad", M, K, N, A, G, dW, db, ws, ws.numel())
    ref = A.T @ G
    assert torch.equal(torch.isnan(dW), torch.isnan(ref)) and torch.equal(dW[torch.isinf(ref)], ref[torch.isinf(ref)])
    assert torch.equal(torch.isinf(db), torch.isinf(G.sum(0)))
    assert _status() == 0
