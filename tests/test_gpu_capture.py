"""Calls on a context's stream while the caller captures it."""

import ctypes as C

import numpy as np
import pytest

import hydrant_gb300 as hy
from hydrant_gb300 import _abi
from tests._harness import camera
from tests.test_gpu_skip import knots, voxels

pytestmark = pytest.mark.gpu


class Capture:
    """Opens and closes a capture through the driver API (relaxed mode)."""

    def __init__(self, ctx):
        self.cuda = C.CDLL("libcuda.so.1")
        self.stream = C.c_void_p(ctx.stream)
        self.ok = None

    def __enter__(self):
        assert self.cuda.cuStreamBeginCapture_v2(self.stream, 2) == 0
        return self

    def __exit__(self, *exc):
        graph = C.c_void_p()
        self.ok = self.cuda.cuStreamEndCapture(self.stream, C.byref(graph)) == 0
        if graph.value:
            self.cuda.cuGraphDestroy(graph)


@pytest.mark.parametrize("warm", [False, True])
def test_batch_refuses_a_capturing_stream(ctx, warm):
    """HY_ERR_STATE, the caller's capture stays valid, and the batch renders
    afterwards as before."""
    torch = pytest.importorskip("torch")
    ctx.set_transfer_fn(knots("first"))
    vol = hy.Volume(ctx, voxels("u8", (64, 64, 64)), 32, 1)
    p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3)
    views = [(hy.camera_view(vol, camera(a=(0.0, 30.0 * i, 2.0))), 48, 40) for i in range(3)]
    b = hy.Batch(ctx, vol, p, views)
    out = torch.zeros(b.nbytes, dtype=torch.uint8, device="cuda")
    host = np.zeros(b.nbytes, np.uint8)
    cfg = _abi.HyBatchConfig()
    torch.cuda.synchronize()
    try:
        if warm:
            b.render_device(out.data_ptr())
        ctx.synchronize()
        lib = hy.lib()
        with Capture(ctx) as cap:
            rcs = (lib.hy_batch_render_device(b.handle, C.c_void_p(out.data_ptr())),
                   lib.hy_batch_render(b.handle, host.ctypes.data_as(C.c_void_p)),
                   lib.hy_batch_autotune(b.handle, C.c_void_p(out.data_ptr()), 1, C.byref(cfg)))
            message = lib.hy_last_error(ctx.handle)
        assert rcs == (_abi.HY_ERR_STATE,) * 3 and b"capturing" in message
        assert cap.ok
        out.zero_()
        torch.cuda.synchronize()
        b.render_device(out.data_ptr())
        ctx.synchronize()
        for img, (view, W, H) in zip(b.split(out.cpu().numpy()), views):
            assert np.array_equal(img, hy.render(ctx, vol, p, view, W, H).rgba)
    finally:
        b.close()
        vol.close()
