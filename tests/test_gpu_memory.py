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
