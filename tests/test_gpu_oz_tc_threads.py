"""pcg_ozaki_gemm_tc from two threads on streams of their own, with operands of different sizes: every
product as if alone (the bar of test_gpu_oz_tc.py), and the flag of each thread's last call."""
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_two_threads():
    from pychem_gb300.scf import ozaki_gemm_tc, ozaki_tc_status
    errors = [[], []]
    start = threading.Barrier(2)

    def work(k, M, N, K):
        g = torch.Generator(device="cuda").manual_seed(k)
        X = torch.randn(M, K, dtype=torch.float64, device="cuda", generator=g)
        Ys = [torch.randn(K, n, dtype=torch.float64, device="cuda", generator=g) for n in (N, N + 64, N)]
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        start.wait()
        outs = []
        with torch.cuda.stream(s):
            for it in range(60):
                Y = Ys[it % 3]
                n = Y.shape[1]
                C = torch.empty(M, n, dtype=torch.float64, device="cuda")
                ozaki_gemm_tc(X, Y, C, M, n, K, K, (n, 1), (n, 1))
                outs.append((Y, C))
            s.synchronize()
            assert ozaki_tc_status("cuda") == 0
            for Y, C in outs:
                scale = X.abs().amax(dim=1, keepdim=True) * Y.abs().amax(dim=0, keepdim=True) * K
                errors[k].append(float(((C - X @ Y).abs() / scale).max()))

    threads = [threading.Thread(target=work, args=a) for a in ((0, 3000, 80, 208), (1, 2500, 96, 300))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(errors[0]) == len(errors[1]) == 60
    assert max(errors[0] + errors[1]) < 1e-12


def test_status_reads_the_last_workspace():
    from pychem_gb300 import scf
    X = torch.randn(130, 40, dtype=torch.float64, device="cuda")
    C = torch.empty(130, 130, dtype=torch.float64, device="cuda")
    scf.ozaki_gemm_tc(X, X, C, 130, 130, 40, 40, (1, 40), (130, 1))
    assert scf.ozaki_tc_status("cuda") == scf.ozaki_tc_status(C.device) == 0
    scf._TC_LAST.by_device[C.device.index][:4] = torch.tensor([3, 0, 0, 0], dtype=torch.uint8, device="cuda")
    assert scf.ozaki_tc_status("cuda") == scf.ozaki_tc_status("cuda:%d" % C.device.index) == 3
    scf.ozaki_gemm_tc(X, X, C, 130, 130, 40, 40, (1, 40), (130, 1))
    assert scf.ozaki_tc_status("cuda") == 0
