"""Leaf kernels of the scaled form: chains of harmonics over eight lanes (P2M,
P2L), evaluation with two or three targets per lane (M2P, L2P), short and long
X / W lists.  Orders at the edges of the chain kernels' instances; split
thresholds whose leaves fall on every pass size (up to 4, 8, 12, 16, 24, 32,
48 targets and more than one pass); a narrow cluster beside a coarse
background gives lists of 1 to hundreds of entries.

The FP64 adaptive solve against the direct sum must stay within five times the
plain form's error on the uniform tree of the same finest cells (V, W and X
pairs are all at least one cell apart, so the truncation errors are of one
size; measured: 0.4 to 1.6 times); a misplaced coefficient would show as an
error of its own size, 1e-2 and more.  The mixed form must stay within its
1e-6 of the FP64 form."""
import numpy as np
import pytest

from laplace_fmm_b200 import FastMultipole3d, InteractionType, compute_exact
from laplace_fmm_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu


def cluster(n, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    src = np.concatenate([0.31 + 0.01 * g.standard_normal((n // 2, 3)), g.random((n - n // 2, 3))])
    return src.clip(0.001, 0.999), g.uniform(-1, 1, n)


@pytest.mark.parametrize("N", [7, 8, 9, 12, 13, 15, 16, 17, 18])
@pytest.mark.parametrize("n,max_leaf,nt", [(3000, 5, 0), (6000, 13, 0), (9000, 40, 1501), (20000, 96, 0)])
def test_leaf_kernels(ctx, N, n, max_leaf, nt):
    src, q = cluster(n, 100 + N)
    tgt = cluster(nt, 7)[0] if nt else None
    args = ((src, q),) if tgt is None else ((src, q), tgt)
    a = FastMultipole3d(*args, N=N, tree_depth=7, max_leaf=max_leaf, ctx=ctx)
    m = FastMultipole3d(*args, N=N, tree_depth=7, max_leaf=max_leaf, precision="mixed", ctx=ctx)
    b = FastMultipole3d(*args, N=N, tree_depth=6, ctx=ctx)
    ex = compute_exact(InteractionType.Force3d, (src, q), tgt)
    assert rel_l2(a.forces, ex) < 5 * rel_l2(b.forces, ex) + 1e-12
    assert rel_l2(m.forces, a.forces) < 1e-6
    s = 0.0 if nt else q * 1e4
    assert rel_l2(m.potentials - s, a.potentials - s) < 1e-6

