"""Entry points that the package itself no longer calls and that callers of the C interface may:
list expansion, pair marking, scattering integrals without prepared factors, and the network's
single-step kernels, against tensor operations.

Tolerances: integrals 2e-12 of the largest (the lanes' bar of test_gpu_eri_lanes.py); FP32
elementwise results 4 roundings (5e-7), sums of M terms M 2^-24 of the sum of magnitudes."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _call(name, *args):
    from pychem_gb300 import _lib
    from pychem_gb300._stream import stream
    return _lib.call(name, *[ctypes.c_void_p(a.data_ptr()) if torch.is_tensor(a) else a for a in args], stream())


def _i32(*v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def test_expand_and_mark():
    bra, ket = _i32(7, 3, 9), _i32(0, 1, 2, 4, 5)
    off = torch.tensor([0, 3, 4, 4], dtype=torch.int64, device="cuda")
    out = torch.full((4, 2), -1, dtype=torch.int32, device="cuda")
    _call("pcg_expand_tasks", 3, bra, ket, off, _i32(1, 2, 0), _i32(1, 0, 0), 4, out)
    assert out.tolist() == [[7, 1], [7, 2], [7, 7], [3, 2]]
    used = torch.zeros(10, dtype=torch.uint8, device="cuda")
    _call("pcg_mark_pairs", torch.cat([out, _i32(9, 9).view(1, 2)]).contiguous(), 5, used)
    assert used.tolist() == [0, 1, 1, 1, 0, 0, 0, 1, 0, 0]


@pytest.mark.parametrize("S", [0.0, 0.7, 9.0])
def test_scattering_without_factors(S):
    from pychem_gb300 import workloads
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.molecule import Molecule
    eng = GpuEngine(Molecule(workloads.water(), "cc-pVDZ")).prepare()
    eng.scattering = S
    eng.schwarz()
    eng.build_tasks()
    eng.compute_eris()
    for cls, rec in eng.classes.items():
        tasks, n = rec["64"]
        want = eng.stores[(cls, "64")]
        got = torch.full_like(want, float("nan"))
        _call("pcg_scattering_class", cls, ctypes.byref(eng.basis_t), ctypes.byref(eng.pairs_t), tasks, n, S, got)
        assert float((got - want).abs().max()) <= 2e-12 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("M,N", [(1, 1), (33, 47), (1000, 65)])
def test_network_steps(M, N):
    g = torch.Generator(device="cuda").manual_seed(M)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    dY, Z = rand(M, N), rand(M, N)
    s = torch.sigmoid(Z.double())
    want = dY.double() * s * (1 + Z.double() * (1 - s))
    _call("pcg_mlp_dsilu", M * N, dY, Z)
    assert float((dY - want).abs().max()) <= 2e-6 * float(want.abs().max())
    db = torch.empty(N, device="cuda")
    _call("pcg_mlp_colsum", M, N, Z, db)
    assert bool(((db - Z.double().sum(0)).abs() <= M * 2.0 ** -24 * Z.double().abs().sum(0)).all())
    Y, T, mask = rand(M, N), rand(M, N), (torch.rand(M, N, device="cuda", generator=g) < 0.6).float()
    out, loss, inv = torch.empty(M, N, device="cuda"), torch.zeros(1, device="cuda"), 1.0 / 7
    _call("pcg_mlp_mse", M * N, Y, T, mask, inv, out, loss)
    d = (Y.double() - T.double()) * mask.double()
    assert float((out - 2 * d * inv).abs().max()) <= 5e-7 * max(1e-30, float(d.abs().max()))
    assert abs(float(loss) - float((d * d).sum() * inv)) <= 1e-5 * float((d * d).sum() * inv) + 1e-12
    w, gr, m, v = rand(M, N), rand(M, N), 0.1 * rand(M, N), rand(M, N).abs()
    wb = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    lr, b1, b2, eps, step = 1e-2, 0.9, 0.999, 1e-8, 3
    m1 = b1 * m.double() + (1 - b1) * gr.double()
    v1 = b2 * v.double() + (1 - b2) * gr.double() ** 2
    w1 = w.double() - lr * (m1 / (1 - b1 ** step)) / ((v1 / (1 - b2 ** step)).sqrt() + eps)
    _call("pcg_mlp_adam", M * N, w, gr, m, v, wb, lr, b1, b2, eps, step)
    # the bias corrections are formed in FP32 from b and step
    assert float((w - w1).abs().max()) <= 5e-5 * lr * float((m1.abs() / v1.sqrt()).max()) * 32 + 5e-7 * float(w1.abs().max())
    assert torch.equal(wb, w.to(torch.bfloat16))
