"""The cache of tuned launch shapes: samples in flight stay with the library's
rule unless the caller sets them, and shapes are kept apart by voxel type."""

import inspect
from types import SimpleNamespace

import hydrant_gb300 as hy
from hydrant_gb300 import _abi, autotune


class FakeBatch:
    def __init__(self):
        self.applied = None

    def set_config(self, *a, **kw):
        b = inspect.signature(hy.Batch.set_config).bind(self, *a, **kw)
        b.apply_defaults()
        self.applied = {k: v for k, v in b.arguments.items() if k != "self"}

    def autotune(self, rgba_ptr, reps):
        return _abi.HyBatchConfig(16, 2, 8, 3, 0, 2)


def test_a_cached_shape_leaves_the_samples_in_flight_to_the_rule(tmp_path):
    path = tmp_path / "cache.json"
    first = autotune.tuned_config(FakeBatch(), "k", 0, path=path)
    assert first["source"] == "autotune" and first["steps_per_iter"] == 2
    batch = FakeBatch()
    again = autotune.tuned_config(batch, "k", 0, path=path)
    assert again["source"] == "cache"
    assert batch.applied == dict(tile_w=16, grab=2, block_warps=8, blocks_per_sm=3, block_queue=0,
                                 steps_per_iter=0)


def test_set_config_defaults_to_the_rule():
    batch = FakeBatch()
    batch.set_config(tile_w=4)
    assert batch.applied["steps_per_iter"] == 0 and batch.applied["tile_w"] == 4


def test_signature_tells_voxel_types_apart():
    params = SimpleNamespace(shader=0, mode=0, composite=0)
    keys = {autotune.signature("gpu", params, _abi.HyVolumeDesc((64, 64, 64), 32, 1, t), [(8, 8)])
            for t in (_abi.DTYPE_U8, _abi.DTYPE_F32)}
    assert len(keys) == 2
