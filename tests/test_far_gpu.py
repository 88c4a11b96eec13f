"""Leaf kernels of the scaled form: chains of harmonics over eight lanes (P2M,
P2L), evaluation with two or three targets per lane (M2P, L2P), short and long
X / W lists; of the plain form; and the 2D power sums.  Orders at the edges of the chain kernels'
instances; split thresholds whose leaves fall on every pass size (up to 4, 8,
12, 16, 24, 32, 48 targets and more than one pass); a narrow cluster beside a
coarse background gives lists of 1 to hundreds of entries.

The FP64 solve's error against the direct sum must fall with the order at
least as fast as the truncation bounds do: a cell's radius is a = sqrt(3)/2 h,
V pairs' centres are 2 h apart, so their bound goes as (a / (2 h - a))^N =
0.764^N, and W and X pairs' as (a / 1.5 h)^N = 0.577^N.  One misplaced
coefficient of degree n would hold the error at the size of the terms of that
degree.  The mixed form must stay within its 1e-6 of the FP64 form."""
import numpy as np
import pytest

from laplace_fmm_b200 import FastMultipole, FastMultipole3d, InteractionType, compute_exact
from laplace_fmm_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu


def cluster(n, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    src = np.concatenate([0.31 + 0.03 * g.standard_normal((n // 2, 3)), g.random((n - n // 2, 3))])
    return src.clip(0.001, 0.999), g.uniform(-1, 1, n)


@pytest.mark.parametrize("n,max_leaf,nt", [(3000, 5, 0), (6000, 13, 0), (9000, 40, 1501), (20000, 96, 0)])
def test_leaf_kernels(ctx, n, max_leaf, nt):
    src, q = cluster(n, 100)
    tgt = cluster(nt, 7)[0] if nt else None
    args = ((src, q),) if tgt is None else ((src, q), tgt)
    ex = compute_exact(InteractionType.Force3d, (src, q), tgt)
    s = 0.0 if nt else q * 1e4
    first = None
    for N in (7, 8, 9, 12, 13, 15, 16, 17, 18):
        a = FastMultipole3d(*args, N=N, tree_depth=7, max_leaf=max_leaf, ctx=ctx)
        m = FastMultipole3d(*args, N=N, tree_depth=7, max_leaf=max_leaf, precision="mixed", ctx=ctx)
        e = rel_l2(a.forces, ex)
        first = first or e
        assert e <= first * 0.764 ** (N - 7), N
        assert rel_l2(m.forces, a.forces) < 1e-6, N
        assert rel_l2(m.potentials - s, a.potentials - s) < 1e-6, N


@pytest.mark.parametrize("N", [1, 4, 9, 16, 18])
@pytest.mark.parametrize("n,depth", [(1, 2), (33, 2), (2048, 2), (1025, 3), (20000, 4)])
def test_plain_leaves(ctx, oracle, N, n, depth):
    """Near field split over a block's warps and gridDim.y, local expansions by
    orders over the warps: few leaves with many targets and the reverse,
    against the CPU restatement at the FP64 parity bar."""
    g = np.random.Generator(np.random.PCG64(n))
    src, q = g.random((n, 3)), g.uniform(0.1, 1, n)
    f = FastMultipole3d((src, q), N=N, tree_depth=depth, ctx=ctx)
    pot, fld = oracle.fmm3d(src, q, N=N, depth=depth)
    assert rel_l2(f.potentials, pot) < 1e-12
    if n > 1:
        assert rel_l2(f.forces, fld) < 1e-12


@pytest.mark.parametrize("N", [1, 2, 8, 9, 16, 17, 25, 30])
@pytest.mark.parametrize("n,depth", [(5, 3), (700, 4), (9001, 5)])
def test_power_sums_2d(ctx, oracle, N, n, depth):
    """The 2D power sums at the edges of their steps of eight orders, leaves of
    a few to more than 32 sources, against the CPU restatement at the FP64
    parity bar."""
    g = np.random.Generator(np.random.PCG64(n + N))
    src, q = g.random((n, 2)), g.uniform(0.1, 1, n)
    f = FastMultipole((src, q), N=N, tree_depth=depth, ctx=ctx)
    pot, fld = oracle.fmm2d(src, q, N=N, depth=depth)
    assert rel_l2(f.potentials, pot) < 1e-12
    assert rel_l2(np.stack([f.forces.real, f.forces.imag], 1), fld) < 1e-12
