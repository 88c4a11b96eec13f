"""Kernels that only large levels reach, on both sides of their lines: the
close lists with a thread per cell (above 131,072 cells in 3D, 16,384 in 2D),
the U / W lists with a thread per leaf (above 131,072 and 16,384 leaves), the
mixed form's M2M on the tensor cores (above 6,144 cells)."""
import numpy as np
import pytest

from helpers import assert_trees_equal, gpu_adaptive_tree, gpu_tree
from laplace_fmm_b200 import FastMultipole3d
from laplace_fmm_b200.workloads import clustered2d, plummer_mix3d, rel_l2, uniform3d
from oracle import adaptive as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,depth,line", [(3, 400000, 7, 131072), (2, 60000, 9, 16384)])
def test_close_lists_of_large_levels(ctx, oracle, dim, n, depth, line):
    """Lists equal to the oracle's in order, on levels below and above the line."""
    g = np.random.Generator(np.random.PCG64(n))
    pts, q = g.random((n, dim)), g.uniform(-1, 1, n)
    a = gpu_tree(ctx, dim, pts, q, depth)
    sizes = [len(lv["code"]) for lv in a["levels"]]
    assert sizes[-1] > line > sizes[-2]
    assert_trees_equal(a, oracle.tree(dim, pts, q, depth, halved=False), n)


@pytest.mark.parametrize("dim,line", [(3, 131072), (2, 16384)])
def test_leaf_lists_of_large_trees(ctx, dim, line):
    """U and W lists of sampled leaves of a tree above the line, against their
    definitions over all cells: U(B) the leaves that touch B, W(B) the finer
    cells that do not touch B and whose parent does."""
    if dim == 3:
        src, q = plummer_mix3d(300000, seed=9)
        cells, lists, _, _ = gpu_adaptive_tree(ctx, src, q, 10, 2)
    else:
        src, q = clustered2d(60000, seed=9)
        cells, lists, _, _ = gpu_adaptive_tree(ctx, src, q, 12, 2, dim=2)
    lev, par, leaf, leaves = cells["level"], cells["parent"], cells["is_leaf"], cells["leaves"]
    assert len(leaves) > line
    top = int(lev.max())
    lo = A._coords(cells["code"], dim) << (top - lev)[:, None]       # corners on the finest grid
    hi = lo + (1 << (top - lev))[:, None]

    def touch(b):
        return ((lo <= hi[b]) & (lo[b] <= hi)).all(axis=1)

    rows = np.random.Generator(np.random.PCG64(1)).choice(len(leaves), 150, replace=False)
    for r in rows:
        b = leaves[r]
        t = touch(b)
        u = np.nonzero(leaf & t)[0]
        np.testing.assert_array_equal(lists["U"][r], u[u != b], err_msg=f"U, leaf {r}")
        w = np.nonzero((lev > lev[b]) & ~t & t[par])[0]
        np.testing.assert_array_equal(lists["W"][r], w, err_msg=f"W, leaf {r}")


@pytest.mark.parametrize("N", [9, 13, 16, 18])
def test_tensor_core_m2m(ctx, N):
    """Level 5 of a uniform depth-7 tree has 32,768 cells that gather their
    children: dense TF32 hi / lo operators in FP32, against the FP64 form.  The
    bar is the one of the tensor-core M2L tests' shifts, half of the mixed
    form's 1e-6."""
    src, q = uniform3d(400000, seed=53)
    a = FastMultipole3d((src, q), N=N, tree_depth=7, precision="mixed", ctx=ctx)
    c = FastMultipole3d((src, q), N=N, tree_depth=7, ctx=ctx)
    assert rel_l2(a.potentials - q * 1e4, c.potentials - q * 1e4) < 5e-7
    assert rel_l2(a.forces, c.forces) < 1e-6
