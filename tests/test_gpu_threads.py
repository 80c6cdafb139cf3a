"""First calls and solves from several threads at the same time."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FIRST = """
import threading, torch
from pychem_gb300.engine import GpuEngine
from pychem_gb300.molecule import Molecule
torch.zeros(1, device="cuda"); torch.cuda.synchronize()
mol = Molecule([["H", 1.0, 0.0, 0.0, 0.0], ["F", 9.0, 0.0, 0.0, 0.92]], "6-31G")
start, out = threading.Barrier(8), [None] * 8
def work(k):
    start.wait()
    eng = GpuEngine(mol).prepare()
    out[k] = (eng.H.cpu(), eng.Q.cpu())
threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
[t.start() for t in threads]; [t.join() for t in threads]
want = GpuEngine(mol).prepare()
for H, Q in out:
    assert torch.equal(H, want.H.cpu()) and torch.equal(Q, want.Q.cpu())
print("ok")
"""


def test_first_calls_of_threads():
    """The tables that the first call of a process makes, from eight threads at once."""
    r = subprocess.run([sys.executable, "-c", FIRST], cwd=REPO, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]


def test_eigensolvers_of_two_threads():
    """Large and small matrices at once, each kernel with its shared memory."""
    import threading
    from pychem_gb300 import eigen
    failed = []

    def work(n, fp32):
        M = torch.randn(2, n, n, dtype=torch.float64, device="cuda")
        A = M + M.transpose(1, 2)
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(200):
                    w, _ = eigen.jacobi(A, fp32=fp32, max_sweeps=1, tol=1e-1)
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            failed.append((n, fp32, e))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in ((136, False), (6, False), (300, True), (12, True))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not failed


def test_solves_of_three_threads():
    """RHF with iteration graphs on streams of their own, one size for each way to the orbitals."""
    import threading
    from pychem_gb300 import workloads
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    from pychem_gb300.scf import rhf
    water = lambda nx, ny, nz: workloads.water_cluster(nx=nx, ny=ny, nz=nz, seed=2)
    mols = [Molecule(water(1, 1, 1), "6-31G"), Molecule(water(2, 2, 1), "6-31G"), Molecule(water(3, 2, 2), "6-31G")]
    want = [rhf(GpuEngine(m).prepare()) for m in mols]
    got = [[], [], []]

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(4):
                got[k].append(rhf(GpuEngine(mols[k]).prepare()))
            torch.cuda.current_stream().synchronize()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for rs, w in zip(got, want):
        assert len(rs) == 4
        for r in rs:
            assert r.converged and abs(r.E - w.E) < 1e-8 and float((r.D - w.D).abs().max()) < 1e-6
