"""The FP32 Gaussian sums do not depend on which exponentials run on the FP32 pipe: a
value below 2^-126 is 0, NaN stays NaN, in every launch shape and at every size."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu

KERNELS = {"gauss2d": (bk.GAUSSIAN, 2), "gaussprod": (bk.GAUSSIAN_PRODUCT_2D, 2),
           "gauss1d": (bk.GAUSSIAN, 1)}
FAR = 200.0


def _points(n, dim):
    return W.SplitMix64(77).normal(n * dim).astype(np.float32).astype(np.float64).reshape(n, dim)


@pytest.mark.parametrize("kernel", KERNELS)
def test_every_shape_flushes_below_the_smallest_normal_number(ctx, kernel):
    """One point repeated over two chunks of 32 references: f = 2^x(q) for exponents x from
    -128 to -124, against shape 0 (all on ex2.approx.ftz): zero at the same queries (one
    step of an FP32 exponent, 2^-17, aside) and within 1e-6 elsewhere: 2.1e-7 of the
    polynomial, 2^-22 of ex2.approx and a few roundings of the sum (the exponents' own
    rounding is shared). The masses are 1: at 1/64 the products are below the smallest
    normal number, where FP32 steps are 2^-17 of a value."""
    kind, dim = KERNELS[kernel]
    x = np.linspace(-128.0, -124.0, 4001)
    q = np.zeros((x.size, dim))
    q[:, 0] = np.sqrt(-2 * x * np.log(2.0))
    ctx.upload(bk.REFERENCE, np.zeros((64, dim)), np.ones(64))
    ctx.upload(bk.QUERY, q)
    desc = bk.kernel_desc(kind, dim, 1.0)
    try:
        out = []
        for v in range(ctx.launch_variants()[0]):
            ctx.set_launch_variant(v)
            out.append(ctx.eval_all(desc, normalized=False))
    finally:
        ctx.set_launch_variant(-1)
    edge = np.abs(x + 126.0) < 2.0 ** -16
    assert np.all(out[0][(x < -126.0) & ~edge] == 0) and np.all(out[0][(x > -126.0) & ~edge] > 0)
    for f in out[1:]:
        np.testing.assert_array_equal(f[~edge] == 0, out[0][~edge] == 0)
        np.testing.assert_allclose(f[~edge], out[0][~edge], rtol=1e-6, atol=0)


@pytest.mark.parametrize("kernel", KERNELS)
def test_every_shape_keeps_a_nan_reference(ctx, kernel):
    kind, dim = KERNELS[kernel]
    desc = bk.kernel_desc(kind, dim, 0.3)
    refs = _points(300, dim)
    ctx.upload(bk.QUERY, refs[:70])
    try:
        for pos in range(32):
            bad = refs.copy()
            bad[64 + pos, dim - 1] = np.nan
            ctx.upload(bk.REFERENCE, bad, np.full(300, 1 / 300))
            for v in range(-1, ctx.launch_variants()[0]):
                ctx.set_launch_variant(v)
                assert np.isnan(ctx.eval_all(desc)).all(), (pos, v)
    finally:
        ctx.set_launch_variant(-1)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("n", [3_000, 20_500])   # the split form; the fixed shape above 3e8 pairs
def test_isolated_points_by_default(ctx, kernel, n):
    """A query out of every reference's reach has density 0, and an isolated point the
    likelihood -inf; a NaN reference makes every density NaN."""
    kind, dim = KERNELS[kernel]
    desc = bk.kernel_desc(kind, dim, 0.05)
    refs = _points(n, dim)
    q = refs.copy()
    q[0] = FAR
    w = np.full(n, 1 / n)
    ctx.upload(bk.REFERENCE, refs, w)
    ctx.upload(bk.QUERY, q)
    f = ctx.eval_all(desc)
    assert f[0] == 0.0 and np.all(f[1:] > 0)
    alone = refs.copy()
    alone[17] = FAR
    ctx.upload(bk.REFERENCE, alone, w)
    assert ctx.likelihood_cv(desc) == -np.inf
    for pos in (4, 9, 14, 31):
        bad = refs.copy()
        bad[pos] = np.nan
        ctx.upload(bk.REFERENCE, bad, w)
        assert np.isnan(ctx.eval_all(desc)).all(), pos
