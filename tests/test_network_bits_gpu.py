"""A network is reproducible from its seeds and rows: gradients and trained parameters
keep the bits that tests/golden/network_bits.npz holds (every 64th parameter, the loss
and the SHA-256 of all of them; recorded when every point was one thread's and every sum
ran in point, feature or partial order)."""
from __future__ import annotations

import hashlib
import os

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "network_bits.npz")


def _rows():
    xy = W.SplitMix64(61).uniform(2 * 30_000, -4, 4).astype(np.float32).astype(np.float64)
    xy = xy.reshape(-1, 2)
    x, y = xy[:, 0], xy[:, 1]
    return xy, 0.5 * x * y + 0.25 * y * y - 0.125 * x


def _check(name, values, loss):
    with np.load(GOLDEN) as g:
        np.testing.assert_array_equal(values[::64], g[name])
        assert loss == float(g[name + "_loss"])
        assert hashlib.sha256(values.tobytes()).digest() == g[name + "_sha"].tobytes()


@pytest.mark.parametrize("engine", [bk.ENGINE_TCGEN05, bk.ENGINE_MMA_SYNC])
@pytest.mark.parametrize("n", [1, 129, 8191, 8193])   # one point; ragged; 64 and 65 partials
def test_gradient_keeps_its_bits(engine, n):
    xy, t = _rows()
    s = bk.Surrogate(0, seed=3)
    s.set_engine(engine)
    g, loss = s.gradient(xy[:n], t[:n])
    _check(f"grad_{engine}_{n}", g, loss)


@pytest.mark.parametrize("engine", [bk.ENGINE_TCGEN05, bk.ENGINE_MMA_SYNC])
@pytest.mark.parametrize("batch", [1000, 8192, 10_000])
def test_training_keeps_its_bits(engine, batch):
    xy, t = _rows()
    s = bk.Surrogate(0, seed=3)
    s.set_engine(engine)
    loss = s.train(xy, t, steps=40, batch=batch, lr=2e-3, lr_final=1e-4, seed=11)
    _check(f"train_{engine}_{batch}", s.params()[0], loss)
