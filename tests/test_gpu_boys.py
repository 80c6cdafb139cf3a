"""Boys orders 0 to 8 of every evaluation, through the drop-in fundamentals, against their series in
extended precision, over the table's grid points, the points between them and the ends of its parts.

Tolerance: half a unit in the last place each for the row's leading term, the last step of its sum, and
the product with the prefactor (1.1e-16 each, up to 3.4e-16 together: 5e-16); above order 2 the downward
recursion adds two roundings an order (2.5e-16)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LD = np.longdouble


def reference(top, T):
    """F_0 .. F_top of T < 60: the ascending series of the highest and downward recursion."""
    t = T.astype(LD)
    e = np.exp(-t)
    term = np.full_like(t, 1.0) / (2 * top + 1)
    acc = term.copy()
    for k in range(1, 400):
        term = term * (2 * t) / (2 * top + 2 * k + 1)
        acc = acc + term
    F = [e * acc]
    for m in range(top, 0, -1):
        F.insert(0, (2 * t * F[0] + e) / (2 * m - 1))
    return np.array(F)


@pytest.mark.parametrize("L", range(9))
def test_boys_orders(L):
    from pychem_gb300 import _lib
    grid = np.arange(0, 48 * 64, 7) / 64.0
    T = np.concatenate([grid, grid + 1 / 128.0, np.random.default_rng(L).uniform(0.0, 47.9, 3000), 10.0 ** np.linspace(-6, 0, 200)])
    if L <= 2:
        T = np.concatenate([T, np.random.default_rng(9).uniform(48.0, 59.0, 300)])
    x = np.sqrt(2.0 * T[T > 1e-13])
    T = 0.5 * (x * x)
    n = len(x)
    pf = 0.79788456080286535588                     # sqrt(2 / pi), the fundamentals' factor
    P, one, U, q = np.zeros((n, 3)), np.ones(n), np.full(n, 1.25), np.zeros((1, 3))
    P[:, 0] = x
    out, R = np.zeros((L + 1, n)), np.zeros((n, 3))
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    assert _lib.load().pcg_two_electron_fundamentals(p(out), p(one), p(U), p(P), p(one), p(one), p(q), p(R), n, 1, 1, 1, L, 0,
                                                     0.0) == 0
    want = reference(L, T) * LD(pf * 1.25)
    err = np.abs((out.astype(LD) / want - 1).astype(np.float64))
    steps = (L - np.arange(L + 1))[:, None] if L > 2 else 0
    assert (err <= 5e-16 + 2.5e-16 * steps).all(), float(err.max())
