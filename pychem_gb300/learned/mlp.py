"""The pair network: 40 -> 256 -> 256 -> 256 -> 29, SiLU, BF16 weights used by the
GEMMs with FP32 accumulation and FP32 master weights for Adam.  Forward and backward
run on the library's kernels (pcg_mlp_*)."""
import ctypes

import numpy as np
import torch

from .. import _lib
from .._stream import stream as _stream
from .blocks import NFEAT, NPARAM

DIMS = [NFEAT, 256, 256, 256, NPARAM]


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


class PairMLP:
    def __init__(self, device="cuda", seed=0, dims=DIMS):
        self.dims = list(dims)
        self.dev = torch.device(device)
        g = torch.Generator().manual_seed(seed)
        self.W, self.b = [], []
        for k in range(len(dims) - 1):
            fan_in = dims[k]
            w = torch.randn(dims[k], dims[k + 1], generator=g) * (2.0 / fan_in) ** 0.5
            if k == len(dims) - 2:
                w *= 0.1
            self.W.append(w.to(self.dev))
            self.b.append(torch.zeros(dims[k + 1], device=self.dev))
        self.refresh_bf16()
        self.mW = [torch.zeros_like(w) for w in self.W]
        self.vW = [torch.zeros_like(w) for w in self.W]
        self.mb = [torch.zeros_like(b) for b in self.b]
        self.vb = [torch.zeros_like(b) for b in self.b]
        self.step_count = 0
        self.mean = torch.zeros(NPARAM, device=self.dev)
        self.std = torch.ones(NPARAM, device=self.dev)

    def refresh_bf16(self):
        self.Wb = [w.to(torch.bfloat16).contiguous() for w in self.W]

    @property
    def nlayers(self):
        return len(self.W)

    def forward(self, X, keep=False):
        """X (M, NFEAT) float32 -> (M, NPARAM) normalised outputs."""
        M, n = X.shape[0], self.nlayers
        A = X.contiguous()
        outs = [torch.empty(M, N, dtype=torch.float32, device=self.dev) for N in self.dims[1:]]
        Z = [torch.empty_like(t) if keep and k < n - 1 else None for k, t in enumerate(outs)]
        ptrs = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() if t is not None else None for t in ts])
        _lib.call("pcg_mlp_forward", n, (ctypes.c_int * (n + 1))(*self.dims), M, _p(A), ptrs(self.Wb), ptrs(self.b),
                  ptrs(outs), ptrs(Z), _stream())
        _lib.launch_count += n
        return outs[-1], list(zip([A] + outs[:-1], Z))

    def backward(self, dY, cache):
        """Gradients (dW, db) per layer for output gradient dY (M, NPARAM)."""
        M = dY.shape[0]
        G = dY.contiguous()
        lib = _lib.load()
        ws = torch.empty(max(lib.pcg_mlp_wgrad_workspace(M, k, n) for k, n in zip(self.dims, self.dims[1:])),
                         dtype=torch.uint8, device=self.dev)
        grads = [None] * self.nlayers
        for k in reversed(range(self.nlayers)):
            K, N = self.dims[k], self.dims[k + 1]
            A = cache[k][0]
            dW = torch.empty(K, N, dtype=torch.float32, device=self.dev)
            db = torch.empty(N, dtype=torch.float32, device=self.dev)
            _lib.call("pcg_mlp_wgrad", M, K, N, _p(A), _p(G), _p(dW), _p(db), _p(ws), ws.numel(), _stream())
            grads[k] = (dW, db)
            if k > 0:
                # dA, times the derivative of the activation below it
                Z = cache[k - 1][1]
                dA = torch.empty(M, K, dtype=torch.float32, device=self.dev)
                _lib.call("pcg_mlp_gemm", M, K, N, _p(G), N, 1, _p(self.Wb[k]), 1, 1, N, _p(dA), K, 0, None, _p(Z),
                          2 if Z is not None else 0, _stream())
                G = dA
        return grads

    def loss_grad(self, Y, T, mask):
        n = Y.numel()
        dY = torch.empty_like(Y)
        loss = torch.zeros(1, dtype=torch.float32, device=self.dev)
        count = mask.sum()
        _lib.call("pcg_mlp_mse_counted", n, _p(Y), _p(T), _p(mask), _p(count), _p(dY), _p(loss), _stream())
        return loss, dY

    def adam(self, grads, lr, b1=0.9, b2=0.999, eps=1e-8):
        self.step_count += 1
        rows = []
        for k, (dW, db) in enumerate(grads):
            rows.append((self.W[k], dW, self.mW[k], self.vW[k], self.Wb[k]))
            rows.append((self.b[k], db, self.mb[k], self.vb[k], None))
        for first in range(0, len(rows), _lib.ADAM_MAX):
            part = rows[first:first + _lib.ADAM_MAX]
            t = _lib.AdamT()
            for j, (w, g, m, v, wb) in enumerate(part):
                t.n[j], t.w[j], t.g[j], t.m[j], t.v[j] = w.numel(), w.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr()
                t.w_bf16[j] = wb.data_ptr() if wb is not None else None
            _lib.call("pcg_mlp_adam_all", len(part), ctypes.byref(t), lr, b1, b2, eps, self.step_count, _stream())

    def predict(self, X):
        Y, _ = self.forward(X)
        return torch.addcmul(self.mean, Y, self.std)

    def check(self):
        """Raises if a tensor-core wait gave up since the last check (its outputs are NaNs);
        synchronises."""
        rc = _lib.load().pcg_mlp_status(_stream())
        if rc:
            raise _lib.PcgError("a wait of the network's GEMM gave up (status %d)" % rc)

    def state(self):
        d = {"dims": np.array(self.dims), "mean": self.mean.cpu().numpy(), "std": self.std.cpu().numpy()}
        for k in range(self.nlayers):
            d["W%d" % k] = self.W[k].cpu().numpy()
            d["b%d" % k] = self.b[k].cpu().numpy()
        return d

    def save(self, path, **extra):
        np.savez_compressed(path, **self.state(), **extra)

    @classmethod
    def load(cls, path, device="cuda"):
        z = np.load(path)
        net = cls(device=device, dims=[int(x) for x in z["dims"]])
        for k in range(net.nlayers):
            net.W[k] = torch.as_tensor(z["W%d" % k], device=net.dev)
            net.b[k] = torch.as_tensor(z["b%d" % k], device=net.dev)
        net.refresh_bf16()
        net.mean = torch.as_tensor(z["mean"], device=net.dev)
        net.std = torch.as_tensor(z["std"], device=net.dev)
        return net
