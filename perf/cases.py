"""The solver's measured workloads: inputs, one pass, its work and its exact results.

Every case goes through a public entry point (``include/lfmm.h`` through the
package's binding, or the package's classes) the way a user's program calls
it: one context kept for the whole program, inputs and outputs in the
program's own buffers, a new solve (tree included) in every pass.  ``kind``
says which entry point:

* ``device``   ``lfmm{2,3}d_solve_device`` / ``..._solve_ex_device`` (max_leaf > 0: adaptive tree)
* ``host``     ``FastMultipole3d(sources, targets)`` on numpy arrays
* ``learned``  ``lfmm3d_solve_learned_device``: leaf size and order from the shipped networks
* ``vector``   ``lfmm3d_solve_vector_device``: charges with three components
* ``batch``    ``lfmm3d_solve_batch_learned_device``: independent problems in one call
* ``plan``     ``lfmm3d_plan_execute``: one geometry, new charges in every pass
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from laplace_fmm_b200 import fmm
from laplace_fmm_b200._lib import AUTO, PRECISION, LfmmLearnedInfo, LfmmSolveOpts, default_context
from laplace_fmm_b200.order import load_params

CLAMP = 1.0e-4          # every distance is at least this (the reference's FORCE_EPS)
EXACT_PAIRS = 1.3e11    # direct sums above this many pairs would take too long


def listed():
    return [
        # the reference's own call on a set so small that launches and host work
        # decide: the inner call of a program that solves thousands of small sets
        dict(name="uniform3d_2k_fp64", kind="device", dim=3, gen="uniform", n=2048, nt=0, N=9, depth=AUTO, max_leaf=0,
             precision="fp64"),
        # the plain FP64 solve of the benchmark's uniform configuration
        dict(name="uniform3d_131k_fp64", kind="device", dim=3, gen="uniform", n=131072, nt=0, N=9, depth=5, max_leaf=0,
             precision="fp64"),
        # a drop-in user of the reference's class: host arrays, sources and
        # separate targets, default tolerance, order and depth
        dict(name="targets3d_60k_host", kind="host", dim=3, gen="uniform", n=60013, nt=20011, N=AUTO, depth=AUTO,
             max_leaf=0, precision="fp64"),
        # clustered set in full precision on the adaptive octree
        dict(name="plummer3d_300k_fp64", kind="device", dim=3, gen="plummer", n=300007, nt=0, N=11, depth=10,
             max_leaf=64, precision="fp64"),
        # mixed form on a small clustered set (the small end of the held-out problems)
        dict(name="gauss3d_10k_mixed", kind="device", dim=3, gen="gauss", n=10007, nt=0, N=14, depth=10, max_leaf=64,
             precision="mixed"),
        # mixed form on a mid-sized clustered set at the accuracy of 1e-6
        dict(name="gauss3d_300k_mixed", kind="device", dim=3, gen="gauss", n=300007, nt=0, N=16, depth=10, max_leaf=64,
             precision="mixed"),
        # the benchmark's headline: 16.8M clustered particles, learned order and leaf size for 1e-6
        dict(name="plummer3d_16m_learned", kind="learned", dim=3, gen="plummer", n=16777216, nt=0, N=16, depth=10,
             max_leaf=AUTO, precision="mixed", tol=1e-6, check=256),
        # vector charges (q x r / r^3), mixed form
        dict(name="plummer3d_1m_vector", kind="vector", dim=3, gen="plummer", n=1048576, nt=0, N=12, depth=10,
             max_leaf=64, precision="mixed"),
        # many uneven problems in one call, each at the order it needs for 1e-6
        dict(name="batch3d_256_learned", kind="batch", dim=3, gen="batch", n=262144, nt=0, count=256, N=14, depth=10,
             max_leaf=AUTO, precision="mixed", tol=1e-6, check=128),
        # iterative solver (boundary elements, time stepping): the same points, new charges
        dict(name="plan3d_300k_mixed", kind="plan", dim=3, gen="plummer", n=300007, nt=0, N=14, depth=10, max_leaf=64,
             precision="mixed"),
        # the benchmark's 2D configuration: 4.2M clustered particles on the adaptive quadtree
        dict(name="clustered2d_4m", kind="device", dim=2, gen="cluster", n=4194304, nt=0, N=21, depth=12, max_leaf=32,
             precision="fp64"),
        # the reference's 2D call with its automatic order and depth
        dict(name="uniform2d_100k", kind="device", dim=2, gen="uniform", n=100003, nt=0, N=AUTO, depth=AUTO,
             max_leaf=0, precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges: sizes log-uniform (odd ones among
    them), orders, leaf sizes and distributions as the programs above meet."""
    kind = rng.choice(["plain", "plain", "host", "adaptive", "mixed", "mixed", "learned", "vector", "batch", "plan",
                       "adaptive2d", "plain2d"])
    c = dict(kind="device", dim=3, gen="uniform", nt=0, N=AUTO, depth=AUTO, max_leaf=0, precision="fp64")
    clustered = rng.choice(["plummer", "gauss", "uniform"])
    if kind == "plain":
        c.update(n=_log_int(rng, 2048, 600000), N=rng.choice([5, 9, 12, 16, AUTO]), nt=rng.choice([0, 0, 1]))
        c["nt"] *= c["n"] // 3 + 1
    elif kind == "host":
        c.update(kind="host", n=_log_int(rng, 2048, 300000), N=rng.choice([9, 14, AUTO]), nt=rng.choice([0, 1]))
        c["nt"] *= c["n"] // 2 + 1
    elif kind == "adaptive":
        c.update(gen=clustered, n=_log_int(rng, 5000, 600000), N=rng.randint(8, 18), depth=10,
                 max_leaf=rng.choice([32, 64, 96]))
    elif kind == "mixed":
        c.update(gen=clustered, n=_log_int(rng, 5000, 8000000), N=rng.randint(8, 17), depth=10,
                 max_leaf=rng.choice([32, 64, 96, 128]), precision="mixed", nt=rng.choice([0, 0, 1]))
        c["nt"] *= c["n"] // 4 + 1
    elif kind == "learned":
        c.update(kind="learned", gen=clustered, n=_log_int(rng, 20000, 8000000), N=16, depth=10, max_leaf=AUTO,
                 precision="mixed", tol=1e-6, check=256)
    elif kind == "vector":
        c.update(kind="vector", gen=clustered, n=_log_int(rng, 10000, 2000000), N=rng.randint(8, 15), depth=10,
                 max_leaf=rng.choice([32, 64, 96]), precision="mixed")
    elif kind == "batch":
        c.update(kind="batch", gen="batch", n=_log_int(rng, 8192, 262144), count=_log_int(rng, 8, 200), N=14, depth=10,
                 max_leaf=AUTO, precision="mixed", tol=1e-6, check=128)
    elif kind == "plan":
        c.update(kind="plan", gen=clustered, n=_log_int(rng, 10000, 4000000), N=rng.randint(8, 17), depth=10,
                 max_leaf=rng.choice([32, 64, 96]), precision="mixed")
    elif kind == "adaptive2d":
        c.update(dim=2, gen=rng.choice(["cluster", "uniform"]), n=_log_int(rng, 5000, 4194304), N=rng.randint(10, 26),
                 depth=12, max_leaf=rng.choice([16, 32, 48]))
    else:
        c.update(dim=2, n=_log_int(rng, 2048, 2000000), N=rng.choice([12, 21, AUTO]), nt=rng.choice([0, 0, 1]))
        c["nt"] *= c["n"] // 3 + 1
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(seed)


def _inside(n, dim, sample):
    """n points of ``sample(k)`` inside the open unit cube."""
    out, have = [], 0
    while have < n:
        p = sample(n - have + (n - have) // 2 + 16)
        p = p[((p > 0) & (p < 1)).all(dim=1)]
        out.append(p)
        have += len(p)
    return torch.cat(out)[:n].contiguous()


def _points(gen, n, dim, g):
    f64 = dict(dtype=torch.float64, device="cuda", generator=g)

    def mixture(centres, sigma):
        k = len(centres)

        def sample(m):
            i = torch.randint(0, k, (m,), device="cuda", generator=g)
            return centres[i] + sigma[i, None] * torch.randn(m, dim, **f64)
        return sample

    if gen == "uniform":
        return torch.rand(n, dim, **f64)
    if gen == "plummer":       # half a Plummer sphere (scale 0.05), half uniform

        def sample(m):
            u = torch.rand(m, **f64).clamp_(1e-12, 1 - 1e-12)
            r = 0.05 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
            v = torch.randn(m, 3, **f64)
            return 0.5 + r[:, None] * v / v.norm(dim=1, keepdim=True)
        return torch.cat([_inside(n // 2, 3, sample), torch.rand(n - n // 2, 3, **f64)])
    if gen == "gauss":         # Gaussian clusters of different widths
        k = 5
        sigma = torch.exp(math.log(0.005) + (math.log(0.2) - math.log(0.005)) * torch.rand(k, **f64))
        return _inside(n, dim, mixture(torch.rand(k, dim, **f64), sigma))
    if gen == "cluster":       # half uniform, half on 64 narrow clusters
        sigma = torch.full((64,), 0.005, dtype=torch.float64, device="cuda")
        return torch.cat([torch.rand(n // 2, dim, **f64),
                          _inside(n - n // 2, dim, mixture(torch.rand(64, dim, **f64), sigma))])
    raise ValueError(gen)


def _sizes(case):
    """The problem sizes of a batch: from 2,048 up to the case's n, spread over the logarithm."""
    lo, hi, k = math.log(2048), math.log(case["n"]), case["count"]
    return [int(round(math.exp(lo + (hi - lo) * (i * 0.6180339887498949 % 1.0)))) | 1 for i in range(k)]


def _inputs(case, seed):
    """(sources, charges, targets or None) on the GPU; batches: problems one after another."""
    g = _gen(seed)
    dim, n = case["dim"], case["n"]
    uni = dict(dtype=torch.float64, device="cuda", generator=g)
    if case["kind"] == "batch":
        parts = []
        for i, m in enumerate(_sizes(case)):
            if i % 2:
                c = 0.2 + 0.6 * torch.rand(1, 3, **uni)
                parts.append(_inside(m, 3, lambda k, c=c: c + 0.05 * torch.randn(k, 3, **uni)))
            else:
                parts.append(torch.rand(m, 3, **uni))
        pos = torch.cat(parts)
    else:
        pos = _points(case["gen"], n, dim, g)
    shape = (len(pos), 3) if case["kind"] == "vector" else (len(pos),)
    q = 2.0 * torch.rand(shape, **uni) - 1.0
    tgt = _points(case["gen"], case["nt"], dim, g) if case["nt"] else None
    return pos, q, tgt


def prepare(case, seed):
    ctx = default_context()
    pos, q, tgt = _inputs(case, seed)
    kind, n = case["kind"], len(pos)
    nout = len(tgt) if tgt is not None else n
    s = dict(case=case, ctx=ctx, stream=torch.cuda.ExternalStream(ctx.stream), pos=pos, q=q, tgt=tgt, n=n, plan=None)
    if kind == "host":
        s.update(pos=pos.cpu().numpy(), q=q.cpu().numpy(), tgt=None if tgt is None else tgt.cpu().numpy())
        return s
    s["opts"] = LfmmSolveOpts(case["N"], case["depth"], case["max_leaf"], PRECISION[case["precision"]],
                              case.get("tol", 1e-8))
    s["pot"] = torch.zeros(nout, dtype=torch.float64, device="cuda")
    s["fld"] = torch.zeros(nout, case["dim"], dtype=torch.float64, device="cuda")
    if kind in ("learned", "batch"):
        s["params"] = torch.from_numpy(load_params(leaf=True)).cuda()
    if kind == "batch":
        s["offsets"] = np.concatenate([[0], np.cumsum(_sizes(case))]).astype(np.uint64)
    if kind == "plan":
        torch.cuda.synchronize()
        s["plan"] = _Plan(ctx, n, pos, q, s["opts"])
    return s


class _Plan:
    """A plan handle that is given back with the state that holds it."""

    def __init__(self, ctx, n, pos, q, opts):
        self.ctx, self.handle = ctx, ctypes.c_void_p()
        ctx.check(ctx.lib.lfmm3d_plan_create(ctx.handle, n, _ptr(pos), _ptr(q), ctypes.byref(opts),
                                             ctypes.byref(self.handle)), "lfmm3d_plan_create")

    def __del__(self):
        if self.handle and self.ctx.handle:
            self.ctx.lib.lfmm3d_plan_destroy(self.handle)


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


# ---------------------------------------------------------------- one pass
def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "host":
        N, depth = case["N"], case["depth"]
        args = ((s["pos"], s["q"]),) if s["tgt"] is None else ((s["pos"], s["q"]), s["tgt"])
        f = fmm.FastMultipole3d(*args, N=N, tree_depth=depth, precision=case["precision"], max_leaf=case["max_leaf"],
                                ctx=ctx)
        return f.potentials, f.forces
    L, h, n, src, q = ctx.lib, ctx.handle, s["n"], _ptr(s["pos"]), _ptr(s["q"])
    nt, tgt, pot, fld = (0 if s["tgt"] is None else len(s["tgt"])), _ptr(s["tgt"]), _ptr(s["pot"]), _ptr(s["fld"])
    opts = ctypes.byref(s["opts"])
    here = torch.cuda.current_stream()
    s["stream"].wait_stream(here)        # the solve runs on the context's stream
    if kind == "learned":
        info = LfmmLearnedInfo()
        st = L.lfmm3d_solve_learned_device(h, n, src, q, nt, tgt, opts, _ptr(s["params"]), case["tol"], case["check"],
                                           pot, fld, ctypes.byref(info), None)
    elif kind == "batch":
        info = LfmmLearnedInfo()
        st = L.lfmm3d_solve_batch_learned_device(h, len(s["offsets"]) - 1, s["offsets"].ctypes.data_as(ctypes.c_void_p),
                                                 src, q, opts, _ptr(s["params"]), case["tol"], case["check"], pot, fld,
                                                 ctypes.byref(info), None)
    elif kind == "vector":
        st = L.lfmm3d_solve_vector_device(h, n, src, q, nt, tgt, opts, fld, None)
    elif kind == "plan":
        st = L.lfmm3d_plan_execute(s["plan"].handle, q, pot, fld)
    elif case["max_leaf"] or case["precision"] == "mixed":
        fn = L.lfmm3d_solve_ex_device if case["dim"] == 3 else L.lfmm2d_solve_ex_device
        st = fn(h, n, src, q, nt, tgt, opts, pot, fld, None)
    else:
        fn = L.lfmm3d_solve_device if case["dim"] == 3 else L.lfmm2d_solve_device
        st = fn(h, n, src, q, nt, tgt, case["N"], case["depth"], 1e-8, PRECISION[case["precision"]], pot, fld, None)
    ctx.check(st, kind)
    here.wait_stream(s["stream"])
    return (s["fld"],) if kind == "vector" else (s["pot"], s["fld"])


# ---------------------------------------------------------------- work, tolerance, exact results
def work(case):
    """Bytes: positions and charges in, potential and field out.  Flops: the
    method's own arithmetic on a uniform tree with the case's leaf size: near
    field (20 flops per pair, 27 or 9 cells' particles per target), the
    rotation form's F(N) (2D: 8 N^2) per far pair with 189 or 27 pairs per
    cell, and one harmonic per coefficient per particle into and out of the
    leaves (8 and 32 flops)."""
    dim, nt = case["dim"], case["nt"]
    n = sum(_sizes(case)) if case["kind"] == "batch" else case["n"]
    out = nt or n
    ncomp = 3 if case["kind"] == "vector" else 1
    N = case["N"] if case["N"] != AUTO else (18 if dim == 3 else 21)
    N = min(N, 18 if dim == 3 else 30)
    leaf = 48.0 if case["max_leaf"] in (0, AUTO) else 0.5 * case["max_leaf"]
    cells = n / leaf * (8.0 / 7.0 if dim == 3 else 4.0 / 3.0)
    if dim == 3:
        F = 2 * sum((k + 1) * (4 * k + 2) for k in range(N)) + 4 * sum(m * m for m in range(1, N + 1)) + 6 * N * (N + 1)
        far, near, coef = 189.0, 27.0, N * (N + 1) / 2
    else:
        F, far, near, coef = 8.0 * N * N, 27.0, 9.0, float(N)
    flops = ncomp * (cells * far * F + coef * (8.0 * n + 32.0 * out)) + 20.0 * near * leaf * out
    points = 0 if case["kind"] == "plan" else dim * (n + nt)
    results = dim * out if case["kind"] == "vector" else (1 + dim) * out
    return {"bytes": 8.0 * (points + ncomp * n + results), "flops": flops}


def tolerance(case):
    """Largest relative difference of another correct form at the same
    precision.  FP64: the parity bar of the tests (the rotation, SIMT and
    tensor-core engines differ by up to 3e-15 here, the spherical and
    Cartesian forms of the harmonics by more); mixed: four times the 2.3e-7 of
    its other engines (SIMT sums carried in FP64); learned solves also choose
    the order and the leaf size, so their truncation errors (each within tol)
    are part of the difference."""
    if case["kind"] in ("learned", "batch"):
        return {"rel": 2.0 * case["tol"]}
    if case["precision"] == "mixed":
        return {"rel": 1.0e-6}
    return {"rel": 1.0e-12}


def _direct(src, q, tgt, skip_self, dim):
    """Direct sums in FP64 with the clamp of the distance: the potential
    (without self terms) and the field of every target."""
    nt, n = len(tgt), len(src)
    pot = torch.zeros(nt, dtype=torch.float64, device=src.device)
    fld = torch.zeros(nt, dim, dtype=torch.float64, device=src.device)
    step = max(1, (1 << 27) // max(1, n))
    qq = q.reshape(n, -1)
    vec = qq.shape[1] == 3
    for a in range(0, nt, step):
        d = [tgt[a:a + step, k, None] - src[None, :, k] for k in range(dim)]
        r2 = sum(x * x for x in d).clamp_(min=CLAMP * CLAMP)
        if dim == 2:
            pr, w = 0.5 * torch.log(r2), r2.reciprocal()
        else:
            pr = r2.rsqrt()
            w = pr / r2
        if skip_self:
            i = torch.arange(len(d[0]), device=src.device)
            pr[i, a + i] = 0.0
        if vec:              # sum of q x d / r^3
            e = [(w * x) @ qq for x in d]
            for k in range(3):
                u, v = (k + 1) % 3, (k + 2) % 3
                fld[a:a + step, k] = e[v][:, u] - e[u][:, v]
            continue
        pot[a:a + step] = pr @ q
        for k in range(dim):
            fld[a:a + step, k] = (w * d[k]) @ q
    if dim == 2:
        fld[:, 1] = -fld[:, 1]           # the conjugate field of the complex form
    return pot, fld


def exact(case, seed):
    """The direct sum of the same inputs: FMM results differ from it by the
    truncation of the expansions and by rounding."""
    sizes = _sizes(case) if case["kind"] == "batch" else [case["n"]]
    if sum(float(m) * (case["nt"] or m) for m in sizes) > EXACT_PAIRS:
        return None
    pos, q, tgt = _inputs(case, seed)
    dim, self_term = case["dim"], (1.0 / CLAMP if case["dim"] == 3 else math.log(CLAMP))
    pots, flds, a = [], [], 0
    for m in sizes:
        src, qs = pos[a:a + m], q[a:a + m]
        pot, fld = _direct(src, qs, src if tgt is None else tgt, tgt is None, dim)
        if tgt is None and qs.dim() == 1:
            pot += qs * self_term        # the reference's self interaction at the clamp
        pots.append(pot)
        flds.append(fld)
        a += m
    pot, fld = torch.cat(pots), torch.cat(flds)
    if case["kind"] == "host":
        return pot.cpu().numpy(), fld.cpu().numpy()
    return (fld,) if case["kind"] == "vector" else (pot, fld)
