"""A wait of the network's GEMM that gave up stops training (the kernel's flag stood in for on the
host)."""
import types

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("flag", [0, 1, 2])
def test_check_raises_when_a_wait_gave_up(monkeypatch, flag):
    from pychem_gb300 import _lib
    from pychem_gb300.learned import mlp
    monkeypatch.setattr(mlp, "_stream", lambda: None)
    monkeypatch.setattr(_lib, "load", lambda: types.SimpleNamespace(pcg_mlp_status=lambda stream: flag))
    net = object.__new__(mlp.PairMLP)
    if flag == 0:
        net.check()
    else:
        with pytest.raises(_lib.PcgError, match="gave up"):
            net.check()
