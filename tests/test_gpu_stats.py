"""hy_render_stats.ms counts every kernel of a render: also those that bring the
skip grid in line with new knots."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from hydrant_gb300 import _abi

pytestmark = pytest.mark.gpu


def test_ms_holds_the_grid_after_new_knots(ctx):
    """Sixteen pixels whose rays miss the volume take a few us, the grid's six
    kernels over 262,144 cells more than twice as long: renders right after
    hy_tf_set report it, repeated ones do not."""
    torch = pytest.importorskip("torch")
    vox = np.zeros((512, 512, 512), np.uint8)
    vox[::8, ::8, ::8] = 200
    vox[:, :, 256:] = 1
    knots = [np.full((9, 4), 0.5, np.float32) for _ in range(2)]
    knots[0][:3, 3] = 0
    knots[1][:4, 3] = 0
    ctx.set_transfer_fn(knots[0])
    vol = hy.Volume(ctx, vox, 64, 1)
    p = hy.shader_params(shader="Volume", sample_rate=0.25, density=0.1)
    away = hy.camera_ptu((3.0, 0.0, 0.0), target=(9.0, 0.0, 0.0))
    view = hy.camera_view(vol, away)
    batch = hy.Batch(ctx, vol, p, [(view, 4, 4)])
    out = torch.zeros(64, dtype=torch.uint8, device="cuda")
    film = torch.zeros(16 * 64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    calls = {
        "render_device": lambda: hy.render_device(ctx, vol, p, view, 4, 4, out.data_ptr()),
        "batch": lambda: batch.render_device(out.data_ptr()),
        "pass": lambda: hy.shade_pass(ctx, vol, p, _abi.PASS_RAY_EMIT, view, film.data_ptr(), 4, 4),
    }
    try:
        for name, call in calls.items():
            ms = {True: [], False: []}
            for i in range(12):
                ctx.set_transfer_fn(knots[i & 1])
                for first in (True, False):
                    call()
                    ms[first].append(ctx.stats().ms)
            first, again = np.median(ms[True][2:]), np.median(ms[False][2:])
            assert first > 2 * again, (name, first, again)
    finally:
        batch.close()
        vol.close()
