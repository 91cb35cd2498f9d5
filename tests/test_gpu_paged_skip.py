"""A realtime pager's march passes over samples without effect through the
cells of its slots and coarse stand-ins: frames along a path with evictions,
bricks drawn coarse, changing knots and prefetched bricks equal the oracle's
given the resident set, sample counts included, from a pool and from gather
textures, below and above the line between the march's forms (155,648 rays on
152 SMs)."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from hydrant_gb300 import _abi
from hydrant_gb300 import workloads as wl
from oracle import oracle as orc
from tests._harness import view_array
from tests.test_gpu_skip import knots, voxels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bs,level,sampler", [
    ("u8", 16, 2, _abi.PAGER_LOADS), ("u8", 16, 2, _abi.PAGER_GATHERS),
    ("u8", 32, 0, _abi.PAGER_GATHERS), ("f32", 16, 1, _abi.PAGER_LOADS)])
@pytest.mark.parametrize("prefetch", [False, True])
def test_frames(ctx, dtype, bs, level, sampler, prefetch):
    torch = pytest.importorskip("torch")
    vox = voxels(dtype, (96, 64, 80))
    vol = hy.Volume(ctx, vox, bs, 1)
    ov = orc.OracleVolume(vox, bs, 1)
    store = hy.Store.from_volume(vol)
    if level:
        store.build_coarse(level)
        ov.build_coarse(level)
    pg = hy.Pager(ctx, store, max(4, vol.info.nonempty // 3), _abi.PAGER_REALTIME, sampler=sampler)
    try:
        path = [hy.camera_orbit((25.0 + 40.0 * f, 30.0, 1.4)) for f in range(5)]
        for f, (cam, tf) in enumerate(zip(path, ("first", "ends", "over", "all", "first"))):
            W, H = ((57, 43), (397, 394))[f % 2]
            ctx.set_transfer_fn(knots(tf))
            p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3, count_samples=True)
            out = torch.zeros(W * H * 4, dtype=torch.uint8, device="cuda")
            pg.render(p, cam, W, H, out.data_ptr())
            samples = ctx.stats().samples
            if prefetch and f + 1 < len(path):
                pg.prefetch(path[f + 1])
            ov.set_present(pg.present())
            op = orc.params_from(p)
            op.lowest_blkcnt = ov.lowest_blkcnt if level else 0
            ref = orc.render(ov, knots(tf), op, view_array(hy.camera_view(pg.volume, cam)), W, H)
            assert np.array_equal(out.cpu().numpy().reshape(H, W, 4), ref["rgba"]), (f, tf)
            assert samples == ref["samples"], (f, tf)
    finally:
        pg.close()
        store.close()
        vol.close()
