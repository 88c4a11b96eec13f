"""The reciprocal square root and the quotient of the near field, refined from
the hardware's approximations, value by value through the solver: one source
and targets in a tree of two levels, where nothing but the near field acts.
Coordinates are integers times a power of two, so r^2 is exact in any order of
its operations."""
import numpy as np
import pytest

from laplace_fmm_b200 import FastMultipole, FastMultipole3d

pytestmark = pytest.mark.gpu
EPS2 = 1e-4 * 1e-4        # the distance clamp
# log2 of the largest coordinate: below, across and above the clamp, up to where
# the tree's box still holds its 1e-7 margin
SCALES = [-30, -12, -4, 0, 7, 22]


def integers(n, dim, bits, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    return np.ldexp(1 + g.random((n, dim)), g.integers(bits - 7, bits, (n, dim))).astype(np.int64) * \
        g.choice([-1, 1], (n, dim))


@pytest.mark.parametrize("scale", SCALES)
def test_reciprocal_square_root(ctx, scale):
    """Potential of a unit charge: 1 / r, off by at most the roundings of x y
    (2^-54) and of the last sum (2^-53) and the series' rest (2^-58)."""
    k = integers(20000, 3, 24, 3)
    tgt = np.ldexp(k.astype(float), scale - 24)
    f = FastMultipole3d((np.zeros((1, 3)), np.ones(1)), tgt, N=4, tree_depth=2, ctx=ctx)
    r2 = (tgt.astype(np.longdouble) ** 2).sum(axis=1)
    ref = 1 / np.sqrt(np.maximum(r2, np.longdouble(EPS2)))
    assert (np.abs(f.potentials - ref) <= (2.0 ** -53 + 2.0 ** -54 + 2.0 ** -58) * ref).all()


@pytest.mark.parametrize("max_leaf", [0, 30000])
@pytest.mark.parametrize("scale", SCALES)
def test_quotient(ctx, scale, max_leaf):
    """x component of the field at targets whose dx is a power of two: exactly
    dx times q / r^2, which must be the correctly rounded quotient but for
    remainders of 2^-72 on the edge between two neighbours.  The charges reach
    past 1e300, where the division takes over."""
    g = np.random.Generator(np.random.PCG64(5))
    k = integers(20000, 1, 24, 4)[:, 0]
    tgt = np.column_stack([np.ldexp(1.0, g.integers(16, 24, len(k)) + scale - 24), np.ldexp(k.astype(float), scale - 24)])
    r2 = np.maximum(tgt[:, 0] ** 2 + tgt[:, 1] ** 2, EPS2)
    for q in (1.0, -0.37, 3.1e-7, 1.7e5, 2.9e303):
        f = FastMultipole((np.zeros((1, 2)), np.array([q])), tgt, N=4, tree_depth=2, max_leaf=max_leaf, ctx=ctx)
        with np.errstate(over="ignore"):
            ref = tgt[:, 0] * (q / r2)
        ok = np.abs(ref) < 1e304       # beyond, the other component may overflow
        got, ref = f.forces.real[ok], ref[ok]
        assert (np.abs(got - ref) <= np.spacing(np.abs(ref))).all()
        assert (got != ref).mean() < 1e-4 if len(ref) else True
