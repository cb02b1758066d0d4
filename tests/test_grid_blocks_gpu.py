"""The grid pipeline's exact fallback on long lists of 16-point tiles, whose 2 x 2 blocks
of flagged tiles are summed as 32-point ones."""
from __future__ import annotations

import numpy as np
import pytest

import bbrcit_kde_b200 as bk
from bbrcit_kde_b200 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _grid(ctx, desc, grid, **cfg):
    out = torch.full((grid[0] * grid[1],), float("nan"), dtype=torch.float64, device="cuda")
    st = ctx.eval_grid(desc, grid, out.data_ptr(), **cfg)
    torch.cuda.synchronize()
    return out.cpu().numpy().reshape(grid[1], grid[0]), st


@pytest.mark.parametrize("nx,ny", [(1009, 1003), (1040, 993), (1008, 1008)])
def test_blocks_are_summed_and_counted(ctx, nx, ny):
    """Bilinear prediction to 0.3%, which enough of the 4,000 tiles miss for blocks to be
    formed (1.5e6 / sqrt(400,000) = 2,372): a tile is exact (1e-5 of the culled sum, which
    both are to 1e-7 and FP32 rounding) or off by more, and the counts are those of the
    exact ones, at ragged right and upper edges and odd numbers of tiles too. Only tiles
    beside an exact one in its 2 x 2 block may be exact without having missed a probe."""
    n = 400_000
    refs = W.config5_refs(n)
    w = np.full(n, 1.0 / n)
    desc = bk.kernel_desc(W.GAUSS, 2, (0.05, 0.05))
    ctx.upload(bk.REFERENCE, refs, mass=w, weight=w)
    ctx.adapt_density_tol(desc, 0.5, rel_tol=1e-6, outputs=False)
    grid = (nx, ny, -4.0, 4.0, -4.0, 4.0)
    want, _ = _grid(ctx, desc, grid, tile=16, cull_rel=1e-7)
    got, st = _grid(ctx, desc, grid, mode=bk.GRID_ANCHORED, tile=16, probes=5, rel_tol=3e-3,
                    low_frac=0.0, cull_rel=1e-7, interp=1)
    assert np.isfinite(got).all()
    ntx, nty = -(-nx // 16), -(-ny // 16)
    assert st.tiles == ntx * nty
    rel = np.zeros((nty * 16, ntx * 16))
    rel[:ny, :nx] = np.abs(got - want) / want
    exact = rel.reshape(nty, 16, ntx, 16).max(axis=(1, 3)) < 1e-5
    points = np.zeros((nty * 16, ntx * 16))
    points[:ny, :nx] = 1
    points = points.reshape(nty, 16, ntx, 16).sum(axis=(1, 3))
    assert st.tiles_flagged == exact.sum() >= 2372
    assert st.tiles_surrogate == st.tiles - exact.sum() > 0
    lattice = (2 * ntx + 1) * (2 * nty + 1)
    assert st.exact_points == lattice + points[exact].sum()
    # whole blocks are among them, and no block has three exact tiles of its four
    full = exact[:nty // 2 * 2, :ntx // 2 * 2].reshape(nty // 2, 2, ntx // 2, 2).sum(axis=(1, 3))
    assert np.any(full == 4) and not np.any(full == 3)


def test_blocks_are_formed_where_they_pay(ctx):
    """Every tile misses a tolerance of 1e-12: 4,032 tiles are enough for blocks with 400,000
    references and not with 20,000, and the values are the exact ones either way."""
    grid = (1009, 1003, -4.0, 4.0, -4.0, 4.0)
    launches = {}
    for n in (20_000, 400_000):
        w = np.full(n, 1.0 / n)
        desc = bk.kernel_desc(W.GAUSS, 2, (0.1, 0.1))
        ctx.upload(bk.REFERENCE, W.config5_refs(n), mass=w, weight=w)
        want, _ = _grid(ctx, desc, grid, tile=32, cull_rel=1e-7)
        cfg = dict(mode=bk.GRID_ANCHORED, tile=16, probes=1, rel_tol=1e-12, low_frac=0.0,
                   cull_rel=1e-7)
        _grid(ctx, desc, grid, **cfg)   # the records and their order are made
        before = ctx.launch_count()
        got, st = _grid(ctx, desc, grid, **cfg)
        launches[n] = ctx.launch_count() - before
        assert st.tiles_flagged == st.tiles == 64 * 63
        np.testing.assert_allclose(got, want, rtol=3e-6, atol=1e-8 * want.max())
    # the list of blocks: the order of the 32-point tiles, two flag kernels, two selections
    assert launches[400_000] >= launches[20_000] + 8, launches
