"""The pair-form culled sum at the edges of its blocks (64 queries), reference tiles
(64) and tile groups (1,024), against the FP64 device path: the skipped part is at
most rel / 2 of every sum and the FP32-compensated arithmetic at most 1e-6 of it
(the direct path's bar), self-sums of the same sizes likewise."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu

KINDS = [(W.GAUSS, 2, (0.3, 0.3)), (W.GAUSS_PROD2D, 2, (0.2, 0.5)), (W.EPAN, 2, (0.8, 0.8)),
         (W.EPAN_PROD2D, 2, (0.9, 0.6)), (W.GAUSS, 1, (0.3, 0.3)), (W.EPAN, 1, (0.6, 0.6))]
SIZES = [(1, 1), (31, 63), (64, 64), (65, 65), (1023, 33), (1025, 129), (4100, 1000)]


def _points(seed, n, dim):
    return W.f32(W.SplitMix64(seed).normal(n * dim).reshape(n, dim))


def _norm(kind, dim, h):
    """Kernel value at distance 0 (Gaussian 1 / (2 pi)^(dim/2), Epanechnikov at most 1)."""
    return 1.0 / (h[0] * (h[1] if dim == 2 else 1.0))


@pytest.mark.parametrize("kind,dim,h", KINDS)
@pytest.mark.parametrize("n,m", SIZES)
def test_edges(ctx, kind, dim, h, n, m):
    refs, q = _points(n, n, dim), _points(m + 7, m, dim)
    rng = W.SplitMix64(5)
    mass, abw = rng.uniform(n, 0.5, 2.0) / n, rng.uniform(n, 0.7, 1.5)
    ctx.upload(bk.REFERENCE, refs, mass=mass, abw=abw)
    ctx.upload(bk.QUERY, q)
    desc = bk.kernel_desc(kind, dim, h)
    want = ctx.eval_all(desc, precision=bk.FP64)
    rel = 1e-6
    got, st = ctx.eval_tol(desc, rel, 0.0)
    # an Epanechnikov value next to the support's edge is a difference from 1, each of
    # its factors off by a few 2^-24: 1e-6 of the largest term of the sum at most
    peak = mass.max() * _norm(kind, dim, h)
    assert np.all(np.abs(got - want) <= (0.5 * rel + 1e-6) * want + 1e-6 * peak)
    assert st.max_bound_ratio <= rel


@pytest.mark.parametrize("n", [1, 63, 65, 1025, 3000])
def test_self_sums(ctx, n):
    refs = _points(n, n, 2)
    w = np.full(n, 1.0 / n)
    desc = bk.kernel_desc(W.GAUSS_PROD2D, 2, (0.3, 0.4))
    ctx.upload(bk.REFERENCE, refs, mass=w, weight=w)
    _, _, exact, _ = ctx.adapt_density(desc, 0.5, precision=bk.FP64)
    _, _, pilot, _ = ctx.adapt_density_tol(desc, 0.5, 1e-6, 0.0)
    np.testing.assert_allclose(pilot, exact, rtol=1.5e-6)
    # new attributes on the same coordinates: the kept order gathers the new masses
    ctx.upload(bk.QUERY, refs)
    want = ctx.eval_all(desc, precision=bk.FP64)
    got, _ = ctx.eval_tol(desc, 1e-6, 0.0)
    np.testing.assert_allclose(got, want, rtol=1.5e-6)
    # other coordinates in the same buffers: a new order
    ctx.upload(bk.REFERENCE, refs[::-1] + 1.0, mass=w, weight=w)
    want = ctx.eval_all(desc, precision=bk.FP64)
    got, _ = ctx.eval_tol(desc, 1e-6, 0.0)
    np.testing.assert_allclose(got, want, rtol=1.5e-6)


def test_not_a_number(ctx):
    """A query that is not a number spoils its own Gaussian sum and no other."""
    refs = _points(3, 500, 2)
    q = _points(4, 200, 2)
    desc = bk.kernel_desc(W.GAUSS, 2, (0.3, 0.3))
    ctx.upload(bk.REFERENCE, refs, mass=np.full(500, 1 / 500))
    ctx.upload(bk.QUERY, q)
    want = ctx.eval_all(desc)
    bad = q.copy()
    bad[:130, 0] = np.nan
    ctx.upload(bk.QUERY, bad)
    got, _ = ctx.eval_tol(desc, 1e-6, 0.0)
    assert np.isnan(got[:130]).all()
    np.testing.assert_allclose(got[130:], want[130:], rtol=2e-6)


@pytest.mark.parametrize("kind,dim", [(W.GAUSS, 1), (W.GAUSS_PROD2D, 2), (W.EPAN, 1)])
@pytest.mark.parametrize("n", [262_144, 262_145, 300_007, 1_100_000, 8_500_000])
@pytest.mark.parametrize("h", [1e-4, 0.02, 5.0])
def test_many_groups(ctx, kind, dim, n, h):
    """More tile groups (1,024 references each) than a block has threads: its scans go over
    the groups in reach -- none, some, more than the list holds (1,074 groups at h = 5) --
    and past 8,192 groups the list is made in two turns. Queries far from all references
    share blocks with others. Bounds as in test_edges; at h = 1e-4 an FP32 coordinate
    (step 2^-22 of a few) is off by 2.4e-3 of a bandwidth in both, the same."""
    refs = W.f32(W.SplitMix64(n).uniform(n * dim, -3.0, 3.0).reshape(n, dim))
    q = W.f32(W.SplitMix64(8).uniform(100 * dim, -3.0, 3.0).reshape(100, dim))
    q[::7] = refs[:15]
    q[50:53] = 40.0
    ctx.upload(bk.REFERENCE, refs, mass=np.full(n, 1.0 / n))
    ctx.upload(bk.QUERY, q)
    desc = bk.kernel_desc(kind, dim, h)
    want = ctx.eval_all(desc, precision=bk.FP64)
    got, st = ctx.eval_tol(desc, 1e-6, 0.0)
    peak = 1.0 / (n * h ** dim)
    # an FP32 exponent of -e is off by e 2^-23 or two of it; below e = 20 that is 1e-5 of one
    # pair's value at most, and sums of many pairs are dominated by near ones
    assert np.all(np.abs(got - want) <= 2e-6 * want + 1e-5 * peak)
    assert st.max_bound_ratio <= 1e-6
