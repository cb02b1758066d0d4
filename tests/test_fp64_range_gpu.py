"""The FP64 Gaussian sums over the range of their masses, and their exponential to a unit
in the last place."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,dim,h", [(W.GAUSS, 2, (0.3, 0.3)), (W.GAUSS_PROD2D, 2, (0.2, 0.5)),
                                        (W.GAUSS, 1, (0.3, 0.3))])
@pytest.mark.parametrize("n,m", [(300, 200), (3000, 40_000)])   # one and four queries a thread
@pytest.mark.parametrize("scale", [1e-290, 1e-70, 1e70, 1e130, 1e200, 1e300])
def test_masses_scale_the_sum(ctx, kind, dim, h, n, m, scale):
    """Masses of any size scale the density; a query out of reach of all has 0. The relative
    error is that of 1e-13 of the sums themselves plus the scaled masses' rounding."""
    rng = W.SplitMix64(n)
    refs, q = rng.normal(n * dim).reshape(n, dim), rng.normal(m * dim).reshape(m, dim)
    mass = rng.uniform(n, 0.5, 2.0) / n
    q[3] = 1e4
    desc = bk.kernel_desc(kind, dim, h)
    ctx.upload(bk.QUERY, q)
    ctx.upload(bk.REFERENCE, refs, mass)
    want = ctx.eval_all(desc, precision=bk.FP64)
    ctx.upload(bk.REFERENCE, refs, mass * scale)
    got = ctx.eval_all(desc, precision=bk.FP64)
    # beyond 1e-308 / 1e-290 of the peak the scaled sums are denormal
    np.testing.assert_allclose(got, want * scale, rtol=1e-13, atol=1e-321)
    assert got[3] == 0.0 and np.all(got[want * scale > 1e-300] > 0)


def test_leave_one_out_with_large_masses(ctx):
    """Masses of 1e200 (a sum that overflows under a bias of 2^512) without the self pair."""
    rng = W.SplitMix64(5)
    x = rng.normal(500).reshape(-1, 1)
    w = np.full(500, 1 / 500)
    desc = bk.kernel_desc(W.GAUSS, 1, 0.4)
    ctx.upload(bk.REFERENCE, x, w, None, w)
    one = ctx.likelihood_cv(desc, bk.FP64)
    ctx.upload(bk.REFERENCE, x, w * 1e200, None, w)
    assert ctx.likelihood_cv(desc, bk.FP64) == pytest.approx(one + 200 * np.log(10), abs=1e-10)


def test_exponential_to_a_unit_in_the_last_place(ctx):
    """One pair of mass 1: exp(s d^2) at the FP64 argument that the kernel forms, against
    exp in extended precision, in units in the last place: half of one for the last sum,
    half for the table's entry, and 0.1 for the polynomial, the reduction and their product
    (|r| <= ln 2 / 32, each off by a few 2^-53 of it)."""
    n = 200_000
    d = np.concatenate([W.SplitMix64(9).uniform(n, 0, 37.0), np.logspace(-12, 1, 2000)])
    ctx.upload(bk.REFERENCE, np.zeros((1, 1)), mass=np.ones(1))
    ctx.upload(bk.QUERY, d.reshape(-1, 1))
    got = ctx.eval_range(bk.kernel_desc(W.GAUSS, 1, 1.0), 0, 0, 0, d.size - 1, normalized=False,
                         precision=bk.FP64)
    x = d * d * -0.5
    want = np.exp(x.astype(np.longdouble))
    ulp = np.spacing(want.astype(np.float64)).astype(np.longdouble)
    assert float(np.max(np.abs(got.astype(np.longdouble) - want) / ulp)) < 1.1
