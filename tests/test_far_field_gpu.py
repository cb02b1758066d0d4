"""Sums to a tolerance leave little out: their error against 64 bits is FP32's own, an order
below the tolerance asked for, although what is left out is always missing."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h", [(8_971, 0.25), (51_330, 0.21), (95_036, 0.23)])
def test_likelihood_to_a_tolerance(ctx, n, h):
    """A 1-D likelihood sums the missing parts of all points. To 1e-6: at most A / 64 of an
    allowance of 1e-6 of the block's smallest sum is left out, 1.6e-8 of each density, and
    the FP32 sums themselves are within 1e-8 on average (their roundings have either sign)."""
    rng = W.SplitMix64(n)
    x = W.f32(np.concatenate([rng.normal(n // 2) * 0.3 - 2.0, rng.normal(n - n // 2) + 2.0]))
    w = rng.uniform(n, 0.5, 1.5)
    w /= w.sum()
    ctx.upload(bk.REFERENCE, x.reshape(-1, 1), w, None, w)
    desc = bk.kernel_desc(W.GAUSS, 1, (h, h))
    want = ctx.likelihood_cv(desc, bk.FP64)
    assert abs(ctx.likelihood_cv_tol(desc, 1e-6, 1e-6) - want) <= 3e-8 * abs(want)
