"""Factored FP64 translations (rot_kernel: rotation blocks and axial blocks on
the FP64 tensor cores) against the per-pair rotation kernels, which apply the
same maps coefficient by coefficient.  Both sum at most N products per
coefficient in each of three steps and up to 189 pairs per cell, so they
differ by about 3 * sqrt(N) * 189 * 2^-53 < 3e-13 of the largest term; the bar
is the parity bar of the FP64 form, 1e-12 (measured: 2e-15)."""
import os

import numpy as np
import pytest

from laplace_fmm_b200 import Context, FastMultipole3d, solve_batch
from laplace_fmm_b200.workloads import rel_l2, uniform3d

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def rotation():
    os.environ["LFMM_M2L"] = "rotation"
    try:
        c = Context(0)
    finally:
        del os.environ["LFMM_M2L"]
    yield c
    c.close()


# orders at the edges of the 4- and 8-wide blocks and of the kernel's
# instances; depths with one ragged tile per class (3), ragged octants and
# sparse slots (4, 5), full 32-target tiles (5 with many particles)
@pytest.mark.parametrize("N", [1, 2, 4, 5, 8, 9, 12, 13, 16, 17, 18])
@pytest.mark.parametrize("n,depth,nt", [(300, 3, 0), (700, 4, 0), (900, 5, 401), (60000, 5, 0)])
def test_factored_translations_match_rotations(ctx, rotation, N, n, depth, nt):
    src, q = uniform3d(n, seed=90 + N)
    args = ((src, q),) if nt == 0 else ((src, q), uniform3d(nt, seed=7)[0])
    a = FastMultipole3d(*args, N=N, tree_depth=depth, ctx=ctx)
    b = FastMultipole3d(*args, N=N, tree_depth=depth, ctx=rotation)
    self_term = 0.0 if nt else q * 1e4
    assert rel_l2(a.potentials - self_term, b.potentials - self_term) < TOL
    assert rel_l2(a.forces, b.forces) < TOL


@pytest.mark.parametrize("N", [3, 8, 12, 14, 16, 17, 18])
@pytest.mark.parametrize("depth", [3, 5])
def test_scaled_translations_match_rotations(ctx, rotation, N, depth):
    """The scaled expansions' translations (axial tables of unit cells, L2L
    added onto the M2L sums): three particles in every cell of the finest grid
    and a split threshold of two make the adaptive tree the uniform one, so
    the two forms differ by rounding (the scaled form's bar, 5e-12) and by the
    plain form's 1e-12 added to every radius, the reference's: in cells of size
    h that moves a point at distance rho from the z axis by 1e-12 r / rho, r and
    rho of the order of h, and so changes the result by about 1e-12 / h, at every
    order (measured: 1e-12 at h = 1/4, 8e-12 at h = 1/16).  N = 17 and 18 once
    differed by 6e-10: an earlier P2M of the scaled form summed only 32 of the
    2 (N - m) columns of an order and lost (16, 0), (17, 0) and (17, 1)."""
    m = 2 ** (depth - 1)
    g = np.random.Generator(np.random.PCG64(N))
    cells = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3).repeat(3, axis=0)
    src = (cells + 0.25 + 0.5 * g.random(cells.shape)) / m
    q = g.uniform(-1, 1, len(src))
    a = FastMultipole3d((src, q), N=N, tree_depth=depth, max_leaf=2, ctx=ctx)
    b = FastMultipole3d((src, q), N=N, tree_depth=depth, ctx=rotation)
    tol = 5e-12 + 1e-12 * m
    assert rel_l2(a.potentials - q * 1e4, b.potentials - q * 1e4) < tol
    assert rel_l2(a.forces, b.forces) < tol


# the low orders' dense FP64 M2L (levels above 512 or 2,048 cells) and the
# factored one below the line, at the orders where the operators' row tiles
# change; the same bar as above
@pytest.mark.parametrize("N", [1, 3, 5, 6, 7, 8])
@pytest.mark.parametrize("n,depth,nt", [(20000, 5, 0), (40000, 5, 3001)])
def test_low_orders_match_rotations(ctx, rotation, N, n, depth, nt):
    src, q = uniform3d(n, seed=50 + N)
    args = ((src, q),) if nt == 0 else ((src, q), uniform3d(nt, seed=8)[0])
    a = FastMultipole3d(*args, N=N, tree_depth=depth, ctx=ctx)
    b = FastMultipole3d(*args, N=N, tree_depth=depth, ctx=rotation)
    self_term = 0.0 if nt else q * 1e4
    assert rel_l2(a.potentials - self_term, b.potentials - self_term) < TOL
    assert rel_l2(a.forces, b.forces) < TOL


@pytest.mark.parametrize("precision,bar", [("fp64", 5e-12), ("mixed", 1e-6)])
@pytest.mark.parametrize("N", [2, 4, 7])
def test_low_orders_in_a_forest(ctx, N, precision, bar):
    """Nine problems of at most 512 finest cells: together their level 3 is above the
    line (dense; FP32 expansions widened and rounded back), alone below it
    (factored).  Bars of the scaled FP64 form and of the mixed form."""
    problems = [uniform3d(4000, seed=60 + k) for k in range(9)]
    kw = dict(N=N, tree_depth=4, max_leaf=2, ctx=ctx)
    for (src, q), (pot, fld) in zip(problems, solve_batch(problems, precision=precision, **kw)):
        b = FastMultipole3d((src, q), **kw)
        assert rel_l2(pot - q * 1e4, b.potentials - q * 1e4) < bar
        assert rel_l2(fld, b.forces) < bar
