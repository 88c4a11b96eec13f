"""tcgen05 engine (hi/lo split, per-slot FP32 flush; the mixed form's M2L on
levels of more than 512 cells from level 4 on, FP16 operands) against the SIMT
FP32 GEMM, the TF32-operand M2L and the FP64 form.  The mixed engines must stay
within the mixed form's 1e-6 of the FP64 form (measured: 2-5e-7).  The other
translations of these trees (M2M up to 6,144 cells, L2L, small levels) run
factored in FP64; the tensor-core M2M of larger levels is in
test_large_levels_gpu.py."""
import os

import pytest

from laplace_fmm_b200 import Context, FastMultipole3d
from laplace_fmm_b200.workloads import plummer_mix3d, rel_l2, uniform3d

pytestmark = pytest.mark.gpu
TOL = 1e-6


def engine_context(name, var="LFMM_M2L"):
    os.environ[var] = name
    try:
        return Context(0)
    finally:
        del os.environ[var]


@pytest.fixture(scope="module")
def tc():
    c = engine_context("tc")
    yield c
    c.close()


@pytest.fixture(scope="module")
def simt():
    c = engine_context("simt")
    yield c
    c.close()


@pytest.fixture(scope="module")
def tf32():
    c = engine_context("tf32", "LFMM_M2L_TYPE")
    yield c
    c.close()


@pytest.fixture(scope="module")
def ldg():
    c = engine_context("ldg", "LFMM_M2L_GATHER")
    yield c
    c.close()


def noself(p, q):
    return p - q * 1e4


@pytest.mark.parametrize("N,depth,gen", [(16, 10, "plummer"), (17, 10, "plummer"), (12, 6, "uniform"),
                                         (15, 6, "uniform")])
def test_f16_and_tf32_operands_agree(tc, tf32, ldg, ctx, N, depth, gen):
    """The FP16 hi/lo M2L (operators and each level's multipoles scaled by
    powers of two into FP16's range, sources split once per level; rows
    brought in by TMA gathers, the default, or by the producers' loads)
    against the TF32 hi/lo M2L: the same 22-bit operand splits, so all land
    equally close to the FP64 form and within a few 1e-7 of each other; the
    two FP16 forms multiply the same staged values (the autotuner may pick
    different slot splits for them, whose partial sums round differently in
    FP32: measured 1.4e-7 apart on the potential)."""
    src, q = (plummer_mix3d if gen == "plummer" else uniform3d)(300000, seed=70 + N)
    kw = dict(N=N, tree_depth=depth, precision="mixed")
    if gen == "plummer":
        kw["max_leaf"] = 64
    a = FastMultipole3d((src, q), ctx=tc, **kw)
    b = FastMultipole3d((src, q), ctx=tf32, **kw)
    c = FastMultipole3d((src, q), ctx=ctx, **{k: v for k, v in kw.items() if k != "precision"})
    ea = rel_l2(noself(a.potentials, q), noself(c.potentials, q))
    eb = rel_l2(noself(b.potentials, q), noself(c.potentials, q))
    fa, fb = rel_l2(a.forces, c.forces), rel_l2(b.forces, c.forces)
    assert ea < TOL and fa < TOL
    assert ea < 1.3 * eb + 1e-8 and fa < 1.3 * fb + 1e-8
    assert rel_l2(noself(a.potentials, q), noself(b.potentials, q)) < 5e-7
    d = FastMultipole3d((src, q), ctx=ldg, **kw)
    assert rel_l2(noself(a.potentials, q), noself(d.potentials, q)) < 3e-7
    assert rel_l2(a.forces, d.forces) < 3e-7


@pytest.mark.parametrize("N", [13, 9, 7, 11, 14, 15, 16])
def test_tc_engine_uniform(tc, simt, ctx, N):
    src, q = uniform3d(262144, seed=40 + N)
    a = FastMultipole3d((src, q), N=N, tree_depth=6, precision="mixed", ctx=tc)
    b = FastMultipole3d((src, q), N=N, tree_depth=6, precision="mixed", ctx=simt)
    c = FastMultipole3d((src, q), N=N, tree_depth=6, ctx=ctx)
    assert rel_l2(noself(a.potentials, q), noself(c.potentials, q)) < TOL
    assert rel_l2(a.forces, c.forces) < TOL
    assert rel_l2(noself(b.potentials, q), noself(c.potentials, q)) < TOL


def test_tc_shifts_keep_fp32_accuracy(tc, ctx):
    """Mixed solves whose M2M and L2L (factored, FP64 on FP32 expansions; dense
    TF32 operators with L2L's diagonal in FP32 before, 3.6e-7, and 1.14e-6 with
    the diagonal in TF32) stay within half of the mixed form's bar."""
    src, q = uniform3d(262144, seed=53)
    a = FastMultipole3d((src, q), N=13, tree_depth=6, precision="mixed", ctx=tc)
    c = FastMultipole3d((src, q), N=13, tree_depth=6, ctx=ctx)
    assert rel_l2(noself(a.potentials, q), noself(c.potentials, q)) < 5e-7


@pytest.mark.parametrize("N", [13, 16])
def test_tc_engine_adaptive(tc, ctx, N):
    src, q = plummer_mix3d(400000, seed=41)
    a = FastMultipole3d((src, q), N=N, tree_depth=10, max_leaf=64, precision="mixed", ctx=tc)
    c = FastMultipole3d((src, q), N=N, tree_depth=10, max_leaf=64, ctx=ctx)
    assert rel_l2(noself(a.potentials, q), noself(c.potentials, q)) < TOL
    assert rel_l2(a.forces, c.forces) < TOL


def test_tc_engine_small_levels_and_targets(tc, ctx):
    """Few cells per level (slot split over several blocks, partial tiles) and
    separate targets."""
    src, q = uniform3d(20000, seed=44)
    tgt, _ = uniform3d(3000, seed=45)
    a = FastMultipole3d((src, q), tgt, N=11, tree_depth=5, precision="mixed", ctx=tc)
    c = FastMultipole3d((src, q), tgt, N=11, tree_depth=5, ctx=ctx)
    assert rel_l2(a.potentials, c.potentials) < TOL
    assert rel_l2(a.forces, c.forces) < TOL


def test_autotuned_split_matches_fixed_rule(ctx):
    """The M2L autotuner only changes how the far slots are split over blocks:
    results within FP32 summation-order differences of the fixed rule
    (measured 1.2e-7)."""
    os.environ["LFMM_M2L_TUNE"] = "0"
    try:
        fixed = Context(0)
    finally:
        del os.environ["LFMM_M2L_TUNE"]
    src, q = plummer_mix3d(300000, seed=47)
    a = FastMultipole3d((src, q), N=13, tree_depth=10, max_leaf=64, precision="mixed", ctx=ctx)
    b = FastMultipole3d((src, q), N=13, tree_depth=10, max_leaf=64, precision="mixed", ctx=fixed)
    assert rel_l2(noself(a.potentials, q), noself(b.potentials, q)) < 5e-7
    assert rel_l2(a.forces, b.forces) < 5e-7
    fixed.close()


@pytest.mark.parametrize("name,var,kept", [("f16", "LFMM_M2L_TYPE", 343 * (6 * 352 + 3 * 160) * 128),
                                           ("tf32", "LFMM_M2L_TYPE", 343 * (11 * 352 + 5 * 160) * 128),
                                           ("simt", "LFMM_M2L", 343 * 272 * 272 * 4)])
def test_operators_kept(name, var, kept):
    """A context keeps the converted operators of an order (N = 18; the SIMT
    engine's of N = 16) and gives the FP64 ones back that they were made from
    (340 MB at N = 18, 203 MB at N = 16)."""
    import torch
    c = engine_context(name, var)
    src, q = uniform3d(30000, seed=3)
    kw = dict(tree_depth=5, precision="mixed", ctx=c)
    FastMultipole3d((src, q), N=7, **kw)
    free = torch.cuda.mem_get_info(0)[0]
    FastMultipole3d((src, q), N=16 if name == "simt" else 18, **kw)
    used = free - torch.cuda.mem_get_info(0)[0]
    c.close()
    assert kept <= used < kept + 120e6
