"""Uploads of every combination of columns, through page-locked memory (up to 64 KB) and as
copies: each column arrives, a missing mass and local bandwidth are 1 and a missing weight is
the mass."""
from __future__ import annotations

import itertools
import threading

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2])
@pytest.mark.parametrize("n", [1, 1300, 2730, 2731, 50_000])
def test_columns(ctx, dim, n):
    rng = W.SplitMix64(n + dim)
    xy = rng.normal(n * dim).reshape(n, dim)
    cols = [rng.uniform(n, 0.5, 2.0) / n for _ in range(3)]
    desc = bk.kernel_desc(W.GAUSS, dim, 0.5)
    for given in itertools.product([False, True], repeat=3):
        mass, abw, weight = (c if g else None for c, g in zip(cols, given))
        ctx.upload(bk.REFERENCE, np.zeros((n, dim)), 3 * cols[1], 3 * cols[2], 3 * cols[0])
        ctx.upload(bk.REFERENCE, xy, mass, abw, weight)
        m, a = ctx.download_attributes()
        want = np.ones(n) if mass is None else mass
        np.testing.assert_array_equal(m, want)
        np.testing.assert_array_equal(a, np.ones(n) if abw is None else abw)
        ctx.unadapt_density()   # the mass becomes the weight
        np.testing.assert_array_equal(ctx.download_attributes()[0],
                                      want if weight is None else weight)
    # the coordinates: the density at the first points, FP64 and FP32 queries
    ctx.upload(bk.REFERENCE, xy, cols[0])
    q = xy[:5]
    ctx.upload(bk.QUERY, np.concatenate([q, xy]))
    d2 = ((q[:, None, :] - xy[None]) ** 2).sum(-1)
    f = np.exp(-2.0 * d2) @ cols[0]
    for precision, tol in ((bk.FP64, 1e-12), (bk.FP32C, 2e-6)):
        got = ctx.eval_range(desc, 0, n - 1, 0, len(q) - 1, normalized=False, precision=precision)
        np.testing.assert_allclose(got, f, rtol=tol)


def test_contexts_of_many_threads_share_no_buffer():
    """Contexts that come and go in eight threads, each with its own small sets: what a
    destroyed one leaves to the next is in use once at a time."""
    errors = []

    def work(seed):
        try:
            for k in range(25):
                rng = W.SplitMix64(1000 * seed + k)
                x = rng.normal(600).reshape(300, 2)
                m = rng.uniform(300, 0.5, 2.0)
                with bk.Context(0) as a, bk.Context(0) as b:
                    for c, shift in ((a, 0.0), (b, 1.0)):
                        c.upload(bk.REFERENCE, x + shift, m)
                        c.upload(bk.QUERY, x[:40] + shift)
                    got = [c.eval_all(bk.kernel_desc(W.GAUSS, 2, 0.5), normalized=False,
                                      precision=bk.FP64) for c in (a, b)]
                    d2 = ((x[:40, None] - x[None]) ** 2).sum(-1)
                    for g in got:
                        np.testing.assert_allclose(g, np.exp(-2.0 * d2) @ m, rtol=1e-11)
                    np.testing.assert_array_equal(a.download_attributes()[0], m)
        except Exception as e:   # reported below, in the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
