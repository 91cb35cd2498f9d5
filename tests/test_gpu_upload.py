"""Volume upload: bricks, means and the chebyshev thumbnail against numpy, at brick
edges on both sides of the line between the kernels' two row orders (padded edges
of 40 and 72), bricks larger than the volume, many and few bricks."""

import numpy as np
import pytest

import hydrant_gb300 as hy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fill", [0.0, 0.01, 0.1, 0.5, 0.95, 1.0])
@pytest.mark.parametrize("grid", [(1, 1, 1), (1, 9, 1), (2, 1, 7), (7, 5, 4), (13, 9, 11)])
def test_chebyshev(ctx, fill, grid):
    """Distance to the nearest brick that is not empty; the largest edge of the
    grid where there is none."""
    gx, gy, gz = grid
    rng = np.random.default_rng(int(fill * 100) + gx)
    full = rng.random((gz, gy, gx)) < fill
    vox = np.repeat(np.repeat(np.repeat(full, 4, 0), 4, 1), 4, 2).astype(np.uint8)
    vol = hy.Volume(ctx, vox, 4, 0)
    try:
        cheb, _ = vol.thumbnails()
        src = np.argwhere(full)
        if len(src):
            at = np.argwhere(np.ones_like(full))
            d = np.abs(at[:, None, :] - src[None]).max(-1).min(-1).reshape(full.shape)
        else:
            d = np.full(full.shape, max(grid))
        assert np.array_equal(cheb, d)
    finally:
        vol.close()
