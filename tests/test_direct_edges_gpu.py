"""The direct sums at the edges of their blocks: the split form of small problems (64
queries, 64 references a warp, 512 a turn of the block) and the FP64 kernel (128-query
blocks, one or four queries a thread) against the FP64 oracle, and the FP64 Gaussian
down to the smallest numbers."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu

KINDS = [(W.GAUSS, 2, (0.3, 0.3)), (W.GAUSS_PROD2D, 2, (0.2, 0.5)), (W.EPAN, 2, (0.8, 0.8)),
         (W.EPAN_PROD2D, 2, (0.9, 0.6)), (W.EPAN_PROD_CONV2D, 2, (0.5, 0.7)),
         (W.GAUSS, 1, (0.3, 0.3)), (W.EPAN, 1, (0.6, 0.6)), (W.EPAN_CONV1D, 1, (0.4, 0.4))]
SIZES = [(1, 1), (63, 65), (64, 64), (65, 127), (511, 129), (513, 63), (4097, 517), (300, 40_000),
         (40_000, 257), (40_000, 385), (20_000, 641), (20_000, 801)]   # FP64: 1, 4, 1, 4 a thread


def _problem(seed, n, m, dim):
    rng = W.SplitMix64(seed)
    refs = W.f32(rng.normal(n * dim).reshape(n, dim))
    q = W.f32(rng.normal(m * dim).reshape(m, dim))
    return refs, q, rng.uniform(n, 0.5, 2.0) / n, rng.uniform(n, 0.7, 1.5)


@pytest.mark.parametrize("kind,dim,h", KINDS)
@pytest.mark.parametrize("n,m", SIZES)
def test_edges(ctx, oracle, kind, dim, h, n, m):
    refs, q, mass, abw = _problem(n + m, n, m, dim)
    ctx.upload(bk.REFERENCE, refs, mass=mass, abw=abw, weight=mass)
    ctx.upload(bk.QUERY, q)
    desc = bk.kernel_desc(kind, dim, h)
    want = oracle.direct(kind, dim, h, refs, mass, q, abw=abw)
    peak = 1.0 / (h[0] * (h[1] if dim == 2 else 1.0)) * mass.max()
    # FP32 products next to the edge of a support are differences from 1, off by 2^-23
    # of the largest term; FP64 ones by 2^-52, n terms rounded each
    got = ctx.eval_all(desc)
    assert np.all(np.abs(got - want) <= 1e-6 * want + 1e-6 * peak)
    got = ctx.eval_all(desc, precision=bk.FP64)
    assert np.all(np.abs(got - want) <= 1e-13 * want + 1e-14 * peak)


@pytest.mark.parametrize("n", [2, 64, 65, 130, 513, 1500])
@pytest.mark.parametrize("precision", [bk.FP32C, bk.FP64])
def test_leave_one_out_edges(ctx, oracle, n, precision):
    refs, _, mass, _ = _problem(n, n, 1, 2)
    mass /= mass.sum()
    ctx.upload(bk.REFERENCE, refs, mass=mass, weight=mass)
    for kind, h in ((W.GAUSS, (0.9, 0.9)), (W.GAUSS_PROD2D, (0.8, 1.1))):
        loo = oracle.self_eval(kind, 2, h, refs, mass, exclude_self=True)
        got = ctx.likelihood_cv(bk.kernel_desc(kind, 2, h), precision)
        assert got == pytest.approx(np.sum(mass * np.log(loo)),
                                    abs=2e-6 if precision == bk.FP32C else 1e-12)


def test_fp64_gaussian_far_values(ctx):
    """exp(-d^2 / 2) down through the denormals to 0, as the library's exp gives it, and
    infinities and NaN as arithmetic treats them. 16 distances per query block share a
    warp with ordinary ones."""
    d = np.array([0.0, 1e-9, 0.5, 5.0, 37.0, 37.6, 37.63, 38.0, 38.4, 38.55, 38.6, 40.0, 42.1, 60.0,
                  1e4, 1e150])
    ctx.upload(bk.REFERENCE, np.zeros((1, 1)), mass=np.ones(1))
    desc = bk.kernel_desc(W.GAUSS, 1, 1.0)
    for sign in (1.0, -1.0):
        ctx.upload(bk.QUERY, (sign * d).reshape(-1, 1))
        got = ctx.eval_range(desc, 0, 0, 0, len(d) - 1, normalized=False, precision=bk.FP64)
        want = np.exp(-0.5 * d * d)
        tiny = 2.0 ** -1073   # two steps of the denormals
        assert np.all(np.abs(got - want) <= 1e-13 * want + tiny), (got, want)
        assert got[-1] == 0.0 and got[-2] == 0.0 and got[-3] == 0.0
    q = np.array([np.inf, -np.inf, np.nan, -np.nan, 1.0])
    ctx.upload(bk.QUERY, q.reshape(-1, 1))
    got = ctx.eval_range(desc, 0, 0, 0, 4, normalized=False, precision=bk.FP64)
    assert got[0] == 0.0 and got[1] == 0.0 and np.isnan(got[2:4]).all()
    assert got[4] == pytest.approx(np.exp(-0.5), rel=1e-15)
    # a thousand far points with large masses add up to nothing
    ctx.upload(bk.REFERENCE, np.full((1000, 1), 100.0), mass=np.full(1000, 1e6))
    assert ctx.eval_range(desc, 0, 999, 4, 4, normalized=False, precision=bk.FP64)[0] == 0.0


@pytest.mark.parametrize("kind,dim,h", KINDS)
@pytest.mark.parametrize("precision", [bk.FP32C, bk.FP64])
def test_every_kernel_is_one_of_the_bandwidths_size(ctx, oracle, kind, dim, h, precision):
    """Local bandwidths of either sign: a kernel value depends on |h a| only (same bounds as
    test_edges)."""
    refs, q, mass, abw = _problem(3, 600, 130, dim)
    abw[::3] *= -1.0
    ctx.upload(bk.REFERENCE, refs, mass=mass, abw=abw, weight=mass)
    ctx.upload(bk.QUERY, q)
    want = oracle.direct(kind, dim, h, refs, mass, q, abw=abw)
    peak = 1.0 / (h[0] * (h[1] if dim == 2 else 1.0)) * mass.max()
    got = ctx.eval_all(bk.kernel_desc(kind, dim, h), precision=precision)
    tol = 1e-6 if precision == bk.FP32C else 1e-13
    assert np.all(np.abs(got - want) <= tol * want + tol * peak)
