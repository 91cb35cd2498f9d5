"""Calls near the limit of device memory: what a call can do without gives way,
and the call succeeds with the same results."""

import pytest

from tests import _limited

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def limited(tmp_path_factory):
    return _limited.build(tmp_path_factory.mktemp("limited"))


UPLOAD = """
import numpy as np
import hydrant_gb300 as hy
from tests._harness import camera
ctx = hy.Context(0)
k = np.random.default_rng(1).random((9, 4)).astype(np.float32); k[:3, 3] = 0
ctx.set_transfer_fn(k)
vox = hy.synth_blobs_u8(3, (96, 96, 96), 9); vox[:, :, :20] = 0; vox[vox == 0] = 1
p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3, count_samples=True)
q = hy.shader_params(shader="Isosurface", mode="Position", sample_rate=0.5, isovalue=0.4)
def images(v):
    view = hy.camera_view(v, camera())
    return [hy.render(ctx, v, s, view, W, H).rgba for s in (p, q) for W, H in ((41, 33), (400, 390))]
def volume(limit):
    start = mem.test_memory_live()
    mem.test_memory_limit(start + limit)
    v = hy.Volume(ctx, vox, 16, 1)
    used = mem.test_memory_live() - start
    mem.test_memory_limit((1 << 64) - 1)
    return v, used
v, used = volume(1 << 40)
want = images(v)
assert v.gather_sampling
v.close()
distances = 12 ** 3 * 16
# room for all but half of the distances: no grid; for all of it: the grid
for limit, full in ((used - distances // 2, False), (used, True)):
    v, now = volume(limit)
    assert v.gather_sampling and (now == used) == full, (now, used)
    for a, b in zip(images(v), want):
        assert np.array_equal(a, b)
    v.close()
print("ok")
"""


def test_upload_without_room_for_its_grid(limited):
    """A volume that fits without the skip grid is uploaded, with its gather
    textures, and renders the same images."""
    assert "ok" in _limited.run(limited, UPLOAD)


DIFF = """
import numpy as np, torch
import hydrant_gb300 as hy
from hydrant_gb300 import fit
from oracle import oracle as orc
from tests.test_gpu_diff_forms import inputs
ctx = hy.Context(0)
cases = []
for n, W, H in ((40, 33, 21), (24, 17, 13), (39, 20, 9), (23, 395, 394), (9, 31, 7)):
    vol, tf, views, va = inputs(ctx, n, 2, 7)
    r = fit.DiffRenderer(ctx, n, views, W, H, 7, density=0.7, ckpt_k=5)
    ref = orc.diff_forward(vol, tf, va, W, H, density=0.7)
    cases.append((r, torch.from_numpy(vol).cuda(), torch.from_numpy(tf).cuda(), ref))
torch.cuda.synchronize()
mem.test_memory_arrays({arrays})
calls = mem.test_memory_array_calls()
# the edges in turn, nothing waited for in between
images = [[r.forward(v, t) for r, v, t, _ in cases] for _ in range(3)]
grads = [r.backward(v, t, 2 * im) for (r, v, t, _), im in zip(cases, images[0])]
torch.cuda.synchronize()
for turn in images:
    for im, (_, _, _, ref) in zip(turn, cases):
        assert np.array_equal(im.cpu().numpy(), ref)
for dv, dt in grads:
    assert torch.isfinite(dv).all() and dv.abs().sum() > 0 and dt.abs().sum() > 0
made = mem.test_memory_array_calls() - calls
print("made", made)
"""


@pytest.mark.parametrize("arrays", [1, 0])
def test_differentiable_edges_in_turn(limited, arrays):
    """Volumes of several edges on one context: one texture, the largest's,
    serves all; without one every call samples by loads (and asks again, but for
    the 9^3 forward, which is over before a texture pays).  The images are the
    oracle's."""
    out = _limited.run(limited, DIFF.format(arrays=arrays))
    assert int(out.split("made")[1]) == (1 if arrays else 17)


FALLBACK = """
import hydrant_gb300 as hy
import tests.test_gpu_diff_forms as forms
mem.test_memory_arrays(0)
ctx = hy.Context(0)
for case in ((23, 2, 17, 13, 5, 1, 1.0), (24, 2, 33, 7, 16, 3, 1.0), (9, 3, 20, 20, 1, 64, 2.0),
             (24, 1, 395, 394, 16, 7, 0.5), (24, 1, 395, 395, 256, 32, 0.5)):
    forms.test_forward_and_gradients(ctx, *case)
forms.test_values_out_of_range(ctx)
print("ok")
"""


def test_differentiable_passes_by_loads(limited):
    """Forward and gradients where the texture cannot be made."""
    assert "ok" in _limited.run(limited, FALLBACK)


FEW_RAYS = """
import numpy as np, torch
import hydrant_gb300 as hy
from hydrant_gb300 import fit
from oracle import oracle as orc
from tests.test_gpu_diff_forms import inputs
ctx = hy.Context(0)
vol, tf, views, va = inputs(ctx, 384, 1, 9)
tv, tt = torch.from_numpy(vol).cuda(), torch.from_numpy(tf).cuda()
for W, H, rate, texture in ((9, 7, 0.25, 0), (40, 33, 0.25, 1), (9, 7, 1.0, 1)):
    r = fit.DiffRenderer(ctx, 384, views, W, H, 9, sample_rate=rate, ckpt_k=7)
    ref = orc.diff_forward(vol, tf, va, W, H, sample_rate=rate)
    calls = mem.test_memory_array_calls()
    mem.test_memory_arrays(texture)
    for keep in (True, False):
        assert np.array_equal(r.forward(tv, tt, keep=keep).cpu().numpy(), ref), (W, rate)
    assert (mem.test_memory_array_calls() > calls) == (texture == 1 and rate < 1), (W, rate)
print("ok")
"""


def test_few_rays_over_a_large_volume(limited):
    """A forward that takes fewer samples than the texture's refresh is worth
    goes by loads and makes none."""
    assert "ok" in _limited.run(limited, FEW_RAYS)


ROOM = """
import numpy as np
import hydrant_gb300 as hy
ctx = hy.Context(0)
k = np.random.default_rng(1).random((9, 4)).astype(np.float32); k[:3, 3] = 0
ctx.set_transfer_fn(k)
vox = np.ones((768, 768, 768), np.uint8)
vox[300:420, 300:420, 300:420] = hy.synth_blobs_u8(3, (120, 120, 120), 9)
p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3)
def volume(limit):
    start = mem.test_memory_live()
    mem.test_memory_limit(start + limit)
    v = hy.Volume(ctx, vox, 64, 1)
    used = mem.test_memory_live() - start
    img = hy.render(ctx, v, p, hy.camera_view(v, hy.camera_orbit((25.0, 65.0, 2.2))), 300, 200).rgba
    v.close()
    mem.test_memory_limit((1 << 64) - 1)
    return used, img
full, want = volume(1 << 40)
distances = 96 ** 3 * 16
# 1 GB of bricks and textures, 20 MB of grid: with 8 MB more, less than a fiftieth is left
less, img = volume(full + (8 << 20))
assert less < full - distances and np.array_equal(img, want), (less, full)
some, img = volume(full + (64 << 20))
assert some == full and np.array_equal(img, want), (some, full)
print("ok")
"""


def test_the_grid_leaves_room(limited):
    """A grid of 20 MB is not taken where it would leave less than a fiftieth of the
    device: the staging buffer of the render after it still fits."""
    assert "ok" in _limited.run(limited, ROOM)
