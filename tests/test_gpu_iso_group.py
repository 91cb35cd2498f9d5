"""Isosurfaces of small launches: a ray's samples on eight lanes and the hits of
a block shaded by one warp.  All modes, images that end inside a block's 8x4
rays, volumes whose rays hit at once (noise), late or not at all, with and
without an apron, against the oracle (the harness's bounds: powf)."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from tests._harness import Case, assert_parity, camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["Color", "Position", "Normal"])
@pytest.mark.parametrize("dtype,bs,pad", [("u8", 16, 1), ("u8", 64, 1), ("u8", 16, 0), ("f32", 32, 1)])
def test_modes(ctx, mode, dtype, bs, pad):
    rng = np.random.default_rng(5)
    vox = hy.synth_blobs_u8(3, (61, 50, 70), 9)
    vox[40:] = rng.integers(0, 256, vox[40:].shape, np.uint8)
    if dtype == "f32":
        vox = vox.astype(np.float32) / np.float32(255)
    c = Case(ctx, vox, bs, pad)
    try:
        for W, H in ((1, 1), (7, 5), (8, 4), (9, 3), (33, 29), (197, 197)):
            for iso, rate in ((0.02, 1.0), (0.6, 0.5), (1.5, 0.5)):
                g, r, _, _ = c.render_both(camera(a=(-50.0, 20.0, 1.9)), W, H, shader="Isosurface",
                                           mode=mode, sample_rate=rate, isovalue=iso)
                assert_parity(g, r, what=f"{mode} {dtype} {bs} {pad} {W}x{H} {iso}")
    finally:
        c.close()
