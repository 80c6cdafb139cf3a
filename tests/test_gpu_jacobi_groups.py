"""Several small matrices to a CTA of the FP64 Jacobi kernel: the launch plan over its whole range
(on the CPU), and batches on both sides of the group sizes with a partial last group.

Tolerances: 1e-12 of the norm and orthogonality 1e-13, the bars of test_gpu_eigen.py."""
import ctypes

import pytest

torch = pytest.importorskip("torch")


def _plan(lib, batch, n):
    p = (ctypes.c_int * 5)()
    assert lib.pcg_jacobi_plan(batch, n, p) == 0
    return list(p)


def test_plan_gives_every_matrix_a_warp():
    from pychem_gb300 import _lib
    lib = _lib.load()
    for n in range(1, 137):
        m = n + (n & 1)
        batches = range(1, 20001) if n <= 32 else list(range(1, 400)) + [1000, 20000, 10 ** 6]
        for batch in batches:
            per, split, rows_per, threads, size = _plan(lib, batch, n)
            assert 1 <= per <= 4 and 32 * per <= threads <= 1024 and threads % 32 == 0
            assert 1 <= split and rows_per * split >= m and size <= 232448 - 1024
    assert lib.pcg_jacobi_plan(1, 137, (ctypes.c_int * 5)()) != 0
    assert max(_plan(lib, b, 4)[0] for b in (455, 456, 912, 5003)) == 4


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 4, 6, 7, 13])
@pytest.mark.parametrize("batch", [456, 913, 3648, 5003, 9729])
def test_grouped_batches(n, batch):
    from pychem_gb300 import eigen
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    M = torch.randn(batch, n, n, dtype=torch.float64, device="cuda", generator=g)
    A = M + M.transpose(1, 2)
    A[1] = torch.diag(torch.arange(n, dtype=torch.float64, device="cuda"))     # nothing to rotate
    A[batch - 1].fill_(1.0)
    w, V = eigen.eigh(A)
    ref = torch.linalg.eigvalsh(A)
    size = ref.abs().amax(dim=1, keepdim=True).clamp_min(1e-30)
    assert float(((w - ref).abs() / size).max()) < 1e-12
    assert float(((A @ V - V * w.unsqueeze(1)).abs() / size.unsqueeze(2)).max()) < 1e-12
    assert float((V.transpose(1, 2) @ V - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max()) < 1e-13
