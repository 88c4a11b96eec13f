"""Separate targets and sources some of whose charges are zero.  A zero charge
puts a source among its leaf's targets (the reference's rule), but outputs exist
for the given targets alone: results against the direct sum, and nothing written
behind the outputs."""
import ctypes

import numpy as np
import pytest

from laplace_fmm_b200 import FastMultipole3d, InteractionType, compute_exact
from laplace_fmm_b200._lib import PRECISION, LfmmSolveOpts
from laplace_fmm_b200.workloads import rel_l2

pytestmark = pytest.mark.gpu


def problem(dim, n, nt, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    src = np.concatenate([g.random((n // 2, dim)), 0.31 + 0.03 * g.standard_normal((n - n // 2, dim))]).clip(0, 1)
    q = g.uniform(-1, 1, n)
    q[g.random(n) < 0.3] = 0.0
    tgt = np.concatenate([g.random((nt // 2, dim)), 0.31 + 0.03 * g.standard_normal((nt - nt // 2, dim))]).clip(0, 1)
    return src, q, tgt


@pytest.mark.parametrize("dim,N,depth,max_leaf,precision,bar", [
    (3, 16, 4, 0, "fp64", 1e-5), (3, 16, 7, 24, "fp64", 1e-5), (3, 16, 7, 24, "mixed", 1e-5), (3, 16, 4, 0, "mixed", 1e-5),
    (2, 24, 5, 0, "fp64", 1e-8), (2, 24, 8, 16, "fp64", 1e-8)])
@pytest.mark.parametrize("n,nt", [(6000, 900), (6000, 7), (300, 2000)])
def test_outputs_of_the_targets_alone(ctx, dim, N, depth, max_leaf, precision, bar, n, nt):
    import torch
    src, q, tgt = problem(dim, n, nt, n + nt)
    pad = n + 64                             # room for a write at any particle's index
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (src, q, tgt)]
    pot = torch.full((nt + pad,), 7.25, dtype=torch.float64, device="cuda")
    fld = torch.full((dim * (nt + pad),), 7.25, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (*d, pot, fld)]
    opts = LfmmSolveOpts(N, depth, max_leaf, PRECISION[precision], 1e-8)
    fn = ctx.lib.lfmm3d_solve_ex_device if dim == 3 else ctx.lib.lfmm2d_solve_ex_device
    ctx.check(fn(ctx.handle, n, p[0], p[1], nt, p[2], ctypes.byref(opts), p[3], p[4], None), "solve")
    ctx.check(ctx.lib.lfmm_check(ctx.handle), "check")
    assert (pot[nt:] == 7.25).all() and (fld[dim * nt:] == 7.25).all()
    kinds = [InteractionType.Potential3d, InteractionType.Force3d] if dim == 3 else \
            [InteractionType.Potential2d, InteractionType.Force2d]
    pe, fe = (compute_exact(k, (src, q), tgt, ctx=ctx) for k in kinds)
    if dim == 2:
        fe = np.stack([fe.real, fe.imag], 1)
    assert rel_l2(pot[:nt].cpu().numpy(), pe) < bar
    assert rel_l2(fld[:dim * nt].cpu().numpy().reshape(nt, dim), fe) < 10 * bar


def test_vector_charges(ctx):
    src, q, tgt = problem(3, 5000, 40, 3)
    g = np.random.Generator(np.random.PCG64(4))
    q3 = g.uniform(-1, 1, (5000, 3)) * (q != 0)[:, None]
    f = FastMultipole3d((src, q3), tgt, N=16, tree_depth=7, max_leaf=24, ctx=ctx)
    E = [compute_exact(InteractionType.Force3d, (src, np.ascontiguousarray(q3[:, c])), tgt, ctx=ctx) for c in range(3)]
    B = np.stack([E[1][:, 2] - E[2][:, 1], E[2][:, 0] - E[0][:, 2], E[0][:, 1] - E[1][:, 0]], axis=1)
    assert rel_l2(f.forces, B) < 1e-4
