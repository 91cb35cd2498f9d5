"""Volume upload: bricks, means and the chebyshev thumbnail against numpy, at brick
edges on both sides of the line between the kernels' two row orders (padded edges
of 40 and 72), bricks larger than the volume, many and few bricks."""

import numpy as np
import pytest

import hydrant_gb300 as hy

pytestmark = pytest.mark.gpu


def bricks_of(vox, bs, pad):
    """(padded bricks, core bricks) of the border-replicated volume, in brick order."""
    g = [-(-d // bs) for d in vox.shape]
    idx = [np.clip(np.arange(-pad, n * bs + pad), 0, d - 1) for n, d in zip(g, vox.shape)]
    full = vox[np.ix_(*idx)]
    out = []
    for z in range(g[0]):
        for y in range(g[1]):
            for x in range(g[2]):
                b = full[z * bs:z * bs + bs + 2 * pad, y * bs:y * bs + bs + 2 * pad,
                         x * bs:x * bs + bs + 2 * pad]
                out.append((b, b[pad:pad + bs, pad:pad + bs, pad:pad + bs]))
    return g, out


@pytest.mark.parametrize("dtype", ["u8", "f32"])
@pytest.mark.parametrize("bs,pad,dims", [
    (1, 0, (5, 4, 3)), (2, 1, (9, 8, 7)), (8, 1, (41, 40, 33)), (16, 2, (50, 17, 33)),
    (38, 1, (80, 40, 39)), (39, 1, (80, 41, 40)), (70, 1, (150, 71, 72)), (71, 1, (150, 72, 73)),
    (128, 1, (200, 130, 129)), (130, 64, (60, 50, 40)), (300, 1, (301, 20, 7))])
def test_bricks_and_means(ctx, dtype, bs, pad, dims):
    rng = np.random.default_rng(bs)
    nx, ny, nz = dims
    vox = rng.integers(1, 256, (nz, ny, nx)).astype(np.uint8)
    vox[rng.random(vox.shape) < 0.3] = 0
    vox[: nz // 2, : ny // 2] = 0
    if dtype == "f32":
        vox = vox.astype(np.float32) * np.float32(0.37) - np.float32(0.1) * (vox > 0)
    vol = hy.Volume(ctx, vox, bs, pad)
    try:
        cheb, mean = vol.thumbnails()
        g, want = bricks_of(vox, bs, pad)
        store = hy.Store.from_volume(vol)
        ne = np.array([b.any() for b, _ in want])
        assert np.array_equal(cheb.ravel() == 0, ne)
        m = np.array([c.astype(np.float64).sum() for _, c in want]) / bs ** 3
        m = m / 255.0 if dtype == "u8" else m
        # f32: sums in another order, float64; then one rounding to float
        assert np.allclose(mean.ravel(), m, rtol=1.2e-7, atol=0)
        for i in np.flatnonzero(ne):
            assert np.array_equal(store.brick(int(i), vox.dtype), want[i][0]), i
        store.close()
    finally:
        vol.close()


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
