"""The factored grid kernels' block forms, each reached by the length of its tile list (148
SMs): 16-point tiles run as lists only as flagged tiles of the pipeline (exact grids and
lattices of 16-point tiles are summed as 32-point ones), clusters of 8, 4 or 2 blocks per
tile up to 444, 888 and 1,776 tiles and one block beyond; 32-point tiles up to 148, 296 and
592, and the tensor cores by themselves from 592 tiles on."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W
from tests.helpers import assert_parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _grid(ctx, desc, grid, **cfg):
    out = torch.full((grid[0] * grid[1],), float("nan"), dtype=torch.float64, device="cuda")
    st = ctx.eval_grid(desc, grid, out.data_ptr(), **cfg)
    torch.cuda.synchronize()
    return out.cpu().numpy(), st


def _direct(ctx, desc, grid):
    nx, ny, x0, x1, y0, y1 = grid
    ctx.upload(bk.QUERY, W.grid_2d(x0, x1, nx, y0, y1, ny))
    return ctx.eval_all(desc)


def _refs(ctx, n=60_000):
    w = np.full(n, 1.0 / n)
    ctx.upload(bk.REFERENCE, W.config5_refs(n), mass=w, weight=w)
    desc = bk.kernel_desc(W.GAUSS, 2, (0.08, 0.08))
    ctx.adapt_density(desc, 0.5, outputs=False)
    return desc


@pytest.mark.parametrize("tx,ty,cut", [(7, 5, 5), (20, 20, 0), (22, 21, 3), (30, 22, 0),
                                       (31, 30, 7), (33, 31, 0)])   # 8, 8, 4, 4, 2, 2 parts
def test_flagged_16_point_tiles(ctx, tx, ty, cut):
    """No tile passes a probe tolerance of 1e-12: all are flagged and summed as 16-point
    tiles (lists below 1,024), the direct sum's values at every point, bitwise again."""
    desc = _refs(ctx)
    grid = (16 * tx - cut, 16 * ty - cut, -4.0, 4.0, -4.0, 4.0)
    want = _direct(ctx, desc, grid)
    cfg = dict(mode=bk.GRID_ANCHORED, tile=16, probes=1, rel_tol=1e-12, low_frac=0.0)
    got, st = _grid(ctx, desc, grid, **cfg)
    assert st.tiles_flagged == st.tiles == tx * ty < 1024
    assert_parity(got, want, 1e-6 + 1e-7, 1e-8, what=f"{tx} x {ty} tiles")
    assert st.max_bound_ratio <= 1e-7
    np.testing.assert_array_equal(_grid(ctx, desc, grid, **cfg)[0], got)


def test_long_list_of_single_16_point_tiles(ctx):
    """2,500 flagged tiles of which no two share a 2 x 2 block, a narrow reference at the
    middle of each over a broad background: one block per tile, most expensive first. The
    narrow ones are below 1% of the background at the probes of neighbouring tiles."""
    g, k = 1600, 50
    dx = 8.0 / g
    rng = W.SplitMix64(12)
    c = -4.0 + (32 * np.arange(k) + 8) * dx
    spikes = np.stack(np.meshgrid(c, c), -1).reshape(-1, 2)
    refs = np.concatenate([rng.uniform(4000, -4.0, 4.0).reshape(-1, 2), spikes])
    mass = np.concatenate([np.full(2000, 1 / 2000), np.full(k * k, 0.1)])
    abw = np.concatenate([np.full(2000, 1.5), np.full(k * k, 0.012)])
    ctx.upload(bk.REFERENCE, refs, mass=mass, abw=abw)
    desc = bk.kernel_desc(W.GAUSS, 2, (1.0, 1.0))
    grid = (g, g, -4.0, 4.0, -4.0, 4.0)
    want = _direct(ctx, desc, grid)
    cfg = dict(mode=bk.GRID_ANCHORED, tile=16, probes=5, rel_tol=2e-2, low_frac=0.0, interp=1)
    got, st = _grid(ctx, desc, grid, **cfg)
    assert st.tiles_flagged == k * k
    exact = np.zeros((g // 16, g // 16), dtype=bool)
    exact[::2, ::2] = True
    inside = np.kron(exact, np.ones((16, 16), dtype=bool)).reshape(-1)
    assert_parity(got[inside], want[inside], 1e-6 + 1e-7, 1e-8, what="single tiles")
    assert np.all(np.abs(got[~inside] / want[~inside] - 1) < 5e-2)
    assert st.max_bound_ratio <= 1e-7
    np.testing.assert_array_equal(_grid(ctx, desc, grid, **cfg)[0], got)


@pytest.mark.parametrize("tx,ty,cut", [(3, 2, 9), (12, 12, 0), (13, 12, 1), (17, 17, 0), (18, 17, 5),
                                       (24, 24, 0), (25, 24, 31)])   # 8, 8, 4, 4, 2, 2, 1 parts
@pytest.mark.parametrize("tile,n", [(16, 60_000), (32, 60_000), (32, 5_000), (32, 1_300)])
def test_exact_grids_in_32_point_tiles(ctx, tx, ty, cut, tile, n):
    """Half as many parts, or one, with fewer than 64 reference tiles (5,000 points); two
    with six of them."""
    desc = _refs(ctx, n)
    grid = (32 * tx - cut, 32 * ty - cut, -4.0, 4.0, -4.0, 4.0)
    want = _direct(ctx, desc, grid)
    got, st = _grid(ctx, desc, grid, tile=tile)
    assert st.exact_points == grid[0] * grid[1]
    assert_parity(got, want, 1e-6 + 1e-7, 1e-8, what=f"{tx} x {ty} tiles")
    assert st.max_bound_ratio <= 1e-7
    np.testing.assert_array_equal(_grid(ctx, desc, grid, tile=tile)[0], got)


@pytest.mark.parametrize("tx,ty,on", [(3, 3, False), (24, 24, False), (37, 16, True),
                                      (25, 24, True)])
def test_tensor_cores_by_themselves_from_one_wave_on(ctx, tx, ty, on):
    """At 1e-5 the automatic setting is bitwise the forced tensor cores from 592 tiles on,
    and bitwise the FP32 pipe below."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (tx * ty >= 4 * sms) == on
    desc = _refs(ctx)
    grid = (32 * tx, 32 * ty, -4.0, 4.0, -4.0, 4.0)
    auto, _ = _grid(ctx, desc, grid, tile=32, cull_rel=1e-5)
    same, _ = _grid(ctx, desc, grid, tile=32, cull_rel=1e-5, tensor_cores=2 if on else 1)
    other, _ = _grid(ctx, desc, grid, tile=32, cull_rel=1e-5, tensor_cores=1 if on else 2)
    np.testing.assert_array_equal(auto, same)
    assert not np.array_equal(auto, other)
