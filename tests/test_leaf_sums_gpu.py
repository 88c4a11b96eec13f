"""P2M of one leaf and P2L of one cell's X list, coefficient by coefficient.

Values: against the Cartesian recurrences in long double.  A coefficient of
degree n is reached in at most N steps of about four rounded operations each,
on terms bounded by |q| r^n (|q| r^-(n+1) irregular), so it is within
8 N u sum |q| r^n, u the unit roundoff.

Sums (FP32): sources at one point with charges that are powers of two have
exactly proportional terms, so their coefficient must be the single source's
value v times the sum of the charges; compensated summation is off by at most
2 u sum |q| |v| (to first order).  Plain FP32 sums of thousands of terms are
off by several times that."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = {0: 2.0 ** -53, 1: 2.0 ** -24}


def leaf_sums(ctx, irregular, N, precision, lists):
    off = np.concatenate([[0], np.cumsum([len(q) for _, q in lists])]).astype(np.uint64)
    x = np.ascontiguousarray(np.concatenate([x for x, _ in lists]))
    q = np.ascontiguousarray(np.concatenate([q for _, q in lists]))
    out = np.zeros(N * (N + 1))
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (off, x, q, out)]
    ctx.check(ctx.lib.lfmm_debug_leaf_sums(ctx.handle, irregular, N, precision, len(lists), *p), "lfmm_debug_leaf_sums")
    return out[0::2] + 1j * out[1::2]


def harmonics(x, N, irregular):
    """conj(B_nm) of every point at row n (n + 1) / 2 + m, long double."""
    X, Y, Z = x.astype(np.longdouble).T
    r2 = X * X + Y * Y + Z * Z
    w = (X + 1j * Y) / (r2 if irregular else 1)
    top = (1 / np.sqrt(r2) if irregular else np.ones_like(r2)).astype(np.clongdouble)
    B = np.zeros((N * (N + 1) // 2, len(X)), dtype=np.clongdouble)
    for m in range(N):
        if m:
            top = -top * w * np.sqrt(np.longdouble(2 * m - 1) / (2 * m))
        below, cur = np.zeros_like(top), top
        for n in range(m, N):
            B[n * (n + 1) // 2 + m] = np.conj(cur)
            d = np.longdouble((n + 1) ** 2 - m * m)
            up = (2 * n + 1) / np.sqrt(d) * Z * cur
            b = np.sqrt(np.longdouble(n * n - m * m) / d)
            below, cur = cur, (up - b * below) / r2 if irregular else up - b * r2 * below
    return B


def sources(irregular, sizes, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    lists = []
    for n in sizes:
        x = g.random((n, 3)) - 0.5
        if irregular:              # a leaf of size 2 whose near face lies one cell away
            c = g.uniform(-1, 1, 3)
            j = g.integers(3)
            c[j] = np.sign(c[j])
            x = 2 * x + 2.5 * c
        lists.append((x.astype(np.float32).astype(float), g.uniform(-1, 1, n).astype(np.float32).astype(float)))
    return lists


# orders at the edges of the kernels' instances and of the chains; counts with
# rests of up to four and eight sources, short and long X lists
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("irregular,sizes", [(0, [1]), (0, [3]), (0, [37]), (0, [96]), (1, [5]), (1, [1, 2, 30, 7]),
                                             (1, [33] * 8), (1, [3, 40, 11] * 20)])
def test_values(ctx, precision, irregular, sizes):
    lists = sources(irregular, sizes, 7 + len(sizes))
    x, q = np.concatenate([a for a, _ in lists]), np.concatenate([b for _, b in lists])
    B = harmonics(x, 18, irregular)
    r = np.linalg.norm(x, axis=1)
    for N in (1, 2, 7, 8, 9, 12, 13, 15, 16, 17, 18):
        got = leaf_sums(ctx, irregular, N, precision, lists)
        k = N * (N + 1) // 2
        n = np.concatenate([np.full(d + 1, d) for d in range(N)])
        size = (np.abs(q) * r ** ((-n[:, None] - 1) if irregular else n[:, None])).sum(axis=1)
        err = np.abs(got - (B[:k] * q).sum(axis=1).astype(complex)) / size
        assert err.max() <= 8 * N * U[precision], (N, err.argmax(), err.max() / U[precision])


@pytest.mark.parametrize("N", [9, 16, 17, 18])
@pytest.mark.parametrize("irregular,sizes", [(0, [32]), (0, [96]), (0, [4000]), (1, [24] * 8), (1, [800] * 4),
                                             (1, [640] * 40)])
def test_fp32_sums_are_compensated(ctx, N, irregular, sizes):
    g = np.random.Generator(np.random.PCG64(N))
    p = np.array([1.37, -0.81, 1.93] if irregular else [0.31, -0.17, 0.43])
    at = lambda n: np.tile(p, (n, 1))
    v = leaf_sums(ctx, irregular, N, 1, [(at(8), np.eye(8)[0])])
    lists = [(at(n), 2.0 ** g.integers(0, 7, n)) for n in sizes]
    Q = sum(q.sum() for _, q in lists)
    err = np.abs(leaf_sums(ctx, irregular, N, 1, lists) - v * Q)
    u = U[1]
    assert (err.real <= 2.02 * u * np.abs(v) * Q * np.sqrt(2)).all(), (err / (np.abs(v) * Q * u + 1e-300)).max()
