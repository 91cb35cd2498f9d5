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


def diff_case(ctx, n=24, seed=4):
    torch = pytest.importorskip("torch")
    from hydrant_gb300 import fit
    from tests.test_gpu_diff_forms import inputs

    vol, tf, views, _ = inputs(ctx, n, 2, 9)
    r = fit.DiffRenderer(ctx, n, views, 33, 21, 9, density=0.7, ckpt_k=5)
    tv, tt = torch.from_numpy(vol).cuda(), torch.from_numpy(tf).cuda()
    img = torch.zeros(2, 21, 33, 4, device="cuda")
    dimg = torch.rand(2, 21, 33, 4, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    dvol, dtf = torch.zeros_like(tv), torch.zeros_like(tt)
    lib = hy.lib()

    def forward():
        ctx.check(lib.hy_diff_forward(
            ctx.handle, C.byref(r.p), C.c_void_p(tv.data_ptr()), C.c_void_p(tt.data_ptr()), r.views,
            r.nviews, r.W, r.H, C.c_void_p(img.data_ptr()), C.c_void_p(r.ckpt.data_ptr()),
            C.c_void_p(r.nsteps.data_ptr())))

    def backward():
        ctx.check(lib.hy_diff_backward(
            ctx.handle, C.byref(r.p), C.c_void_p(tv.data_ptr()), C.c_void_p(tt.data_ptr()), r.views,
            r.nviews, r.W, r.H, C.c_void_p(dimg.data_ptr()), C.c_void_p(r.ckpt.data_ptr()),
            C.c_void_p(r.nsteps.data_ptr()), C.c_void_p(dvol.data_ptr()), C.c_void_p(dtf.data_ptr())))

    return forward, backward, img, dvol, dtf, tv, (r, tt, dimg)


@pytest.mark.parametrize("warm", [False, True])
def test_captured_differentiable_passes(warm):
    """Forward and adjoint are captured on a fresh context and on one that has
    its texture, and replay what the calls give, also after the context has
    rendered a volume of another edge and after the voxels changed."""
    torch = pytest.importorskip("torch")
    ctx = hy.Context(0)
    forward, backward, img, dvol, dtf, tv, keep = diff_case(ctx)
    torch.cuda.synchronize()
    if warm:
        forward()
        backward()
    ctx.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(ctx.stream)):
        forward()
        backward()
    other = diff_case(ctx, 40)
    torch.cuda.synchronize()
    other[0]()
    other[1]()
    ctx.synchronize()
    for scale in (1.0, 0.5):
        tv *= scale
        torch.cuda.synchronize()
        img.zero_(), dvol.zero_(), dtf.zero_()
        torch.cuda.synchronize()
        forward()
        backward()
        ctx.synchronize()
        want = [t.clone() for t in (img, dvol, dtf)]
        img.zero_(), dvol.zero_(), dtf.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(img, want[0])
        # float atomics in another order: 24^3 x 2 views of some 100 samples a ray
        for a, b in zip((dvol, dtf), want[1:]):
            assert torch.linalg.norm((a - b).double()) <= 1e-5 * torch.linalg.norm(b.double())
    del g
    ctx.close()
