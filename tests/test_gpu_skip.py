"""The Volume and Isosurface marches where samples without effect are passed over, in each of
its forms (eight lanes a ray, four or two samples in flight, one at a time),
against the oracle, which takes every sample: images and sample counts equal,
bit for bit.

The image sizes lie on both sides of the lines between the forms (2 and 8 warps
of rays a scheduler on 152 SMs: 38,912 and 155,648 rays); the knots have
transparent runs at the start, inside, at the end, or none, and cases that
must not be passed over (opacities that leave [0, 1], colours that are not
finite where the opacity is zero)."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from hydrant_gb300 import workloads as wl
from oracle import oracle as orc
from tests._harness import Case, assert_parity, camera, view_array

pytestmark = pytest.mark.gpu

SIZES = [(31, 17), (193, 201), (195, 200), (395, 394), (397, 401)]
INF = float("inf")


def knots(name):
    rng = np.random.default_rng(11)
    k = rng.uniform(0.1, 1.0, (7, 4)).astype(np.float32)
    if name == "readme":
        return wl.TF9
    if name == "first":
        k[0] = 0
    elif name == "inside":
        k[2:5, 3] = 0
    elif name == "ends":
        k[:2, 3] = 0
        k[5:, 3] = 0
    elif name == "all":
        k[:, 3] = 0
    elif name == "over":      # v.w passes 1: nothing may be left out
        k[:2, 3] = 0
        k[4, 3] = 3.0
    elif name == "negative":
        k[:2, 3] = 0
        k[4, 3] = -0.5
    elif name == "infinite":  # 0 * inf
        k[1:4, 3] = 0
        k[2, 0] = INF
    return k


def voxels(dtype, dims, seed=3):
    """Blobs with an empty half and a saturated block: free cells, mixed cells
    and empty bricks."""
    v = hy.synth_blobs_u8(seed, dims, 9)
    v[:, :, : dims[0] // 3] = 0
    z, y = dims[2] // 2, dims[1] // 2
    v[z:, y:, -12:] = 255
    if dtype == "u8":
        return v
    return (v.astype(np.float32) * np.float32(1 / 200) - np.float32(0.1)) * (v > 0)


def check_nan(c, cam, W, H, what, **kw):
    """check() for images that hold NaN (equal to itself here)."""
    p = hy.shader_params(count_samples=True, **kw)
    view = hy.camera_view(c.vol, cam)
    g = hy.render(c.ctx, c.vol, p, view, W, H, want_v=True)
    r = orc.render(c.ov, c.tf, orc.params_from(p), view_array(view), W, H)
    assert np.isnan(r["v"]).any(), what
    assert np.array_equal(g.v, r["v"], equal_nan=True), what
    assert np.array_equal(g.rgba, r["rgba"]) and g.samples == r["samples"], what


def check(c, cam, W, H, what, **kw):
    g, r, _, _ = c.render_both(cam, W, H, **kw)
    s = assert_parity(g, r, what=what)
    assert s["max_lsb"] == 0 and s["max_abs"] == 0.0, (what, s)


@pytest.mark.parametrize("wh", SIZES)
@pytest.mark.parametrize("dtype", ["u8", "f32"])
@pytest.mark.parametrize("pad", [1, 0])
def test_sizes(ctx, wh, dtype, pad):
    c = Case(ctx, voxels(dtype, (70, 61, 52)), 32, pad)
    try:
        for rate in (0.25, 1.0):
            check(c, camera(), *wh, f"{wh} {dtype} pad{pad} rate{rate}", shader="Volume",
                  sample_rate=rate, density=0.2)
    finally:
        c.close()


@pytest.mark.parametrize("tf", ["readme", "first", "inside", "ends", "all", "over", "negative",
                                "infinite"])
@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_knots(ctx, tf, dtype):
    c = Case(ctx, voxels(dtype, (64, 48, 40)), 16, 1, tf=knots(tf))
    try:
        for wh in ((37, 29), (200, 210), (400, 399)):
            for composite in (False, True):
                kw = dict(shader="Volume", sample_rate=0.5, density=0.4, composite=composite)
                if tf in ("over", "negative", "infinite"):
                    kw["density"] = 1.0
                if composite and tf == "infinite":
                    continue
                (check_nan if tf == "infinite" else check)(
                    c, camera(a=(-50.0, 20.0, 1.9)), *wh, f"{tf} {dtype} {wh} {composite}", **kw)
    finally:
        c.close()


@pytest.mark.parametrize("iso", [0.0, 1e-6, 0.05, 0.5, 1.0, 1.2, -0.05, -0.2, INF, float("nan")])
@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_isosurface(ctx, iso, dtype):
    """Isovalues on both sides of 0 (the crossing test turns round there), at
    and beyond the voxels' range, in the march's three forms (8 and 24 warps
    of rays a scheduler: 155,648 and 466,944 rays) and composited."""
    if dtype == "u8" and iso < 0:
        pytest.skip("u8 voxels are never negative: every sample crosses, as at 0")
    c = Case(ctx, voxels(dtype, (64, 48, 40)), 16, 1)
    try:
        for wh in ((37, 29), (394, 395), (395, 396), (700, 680)):
            for composite in (False, True):
                if composite and wh[0] > 300:
                    continue
                g, r, _, _ = c.render_both(camera(a=(-50.0, 20.0, 1.9)), *wh, shader="Isosurface",
                                           mode="Position", sample_rate=0.5, isovalue=iso,
                                           composite=composite)
                s = assert_parity(g, r, what=f"iso{iso} {dtype} {wh} {composite}")
                assert s["max_lsb"] == 0 and s["max_abs"] == 0.0, s
    finally:
        c.close()


@pytest.mark.parametrize("dtype,pad", [("u8", 1), ("u8", 0), ("f32", 1)])
def test_small_isosurfaces(ctx, dtype, pad):
    """Isosurfaces with a ray's samples on eight lanes, up to the size where
    they no longer are (2 warps of rays a scheduler: 38,912 rays), with and
    without a surface in reach, and bricks the rays leap over."""
    c = Case(ctx, voxels(dtype, (64, 48, 40)), 16, pad)
    try:
        for wh in ((1, 1), (9, 2), (37, 29), (197, 197), (198, 197)):
            for iso, rate in ((0.4, 1.0), (0.05, 0.25), (0.97, 0.5), (-0.1, 0.5)):
                check(c, camera(a=(-50.0, 20.0, 1.9)), *wh, f"{dtype} {pad} {wh} {iso}",
                      shader="Isosurface", mode="Position", sample_rate=rate, isovalue=iso)
    finally:
        c.close()


def test_brick_edges_and_axis_aligned_rays(ctx):
    """Brick edges that are no power of two and cameras along the axes (step
    components that are zero)."""
    for bs, dims in ((8, (40, 24, 33)), (24, (50, 49, 47)), (40, (81, 40, 79)), (128, (90, 70, 60))):
        c = Case(ctx, voxels("u8", dims), bs, 1)
        try:
            for p in ((2.2, 0.0, 0.0), (0.0, 0.0, -2.2), (0.1, 0.2, 0.05)):
                cam = camera("ptu", a=p, target=(-p[0], 0.0, -p[2]))
                for wh in ((41, 23), (225, 200), (401, 391)):
                    check(c, cam, *wh, f"bs{bs} {p} {wh}", shader="Volume", sample_rate=0.5,
                          density=0.05)
                    check(c, cam, *wh, f"bs{bs} {p} {wh} iso", shader="Isosurface",
                          mode="Position", sample_rate=0.5, isovalue=0.4)
        finally:
            c.close()


@pytest.mark.parametrize("steps", [0, 1, 2])
def test_batch_follows_the_knots(ctx, steps):
    """A batch whose knots change between renders, from transparent runs to
    none and back, equals the per-view images, at both sizes of batch."""
    c = Case(ctx, voxels("u8", (70, 61, 52)), 32, 1)
    try:
        for sizes in (((60, 50), (33, 71)), ((410, 400), (64, 64))):
            p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3)
            views = [(hy.camera_view(c.vol, camera(a=(20.0 * i, 30.0, 2.0))), W, H)
                     for i, (W, H) in enumerate(sizes)]
            b = hy.Batch(ctx, c.vol, p, views)
            try:
                b.set_config(steps_per_iter=steps)
                for tf in ("first", "all", "over", "ends", "first"):
                    ctx.set_transfer_fn(knots(tf))
                    c.tf = knots(tf)
                    imgs = b.render()
                    for (view, W, H), img in zip(views, imgs):
                        one = hy.render(ctx, c.vol, p, view, W, H)
                        assert np.array_equal(img, one.rgba), (tf, W, H)
                        check(c, camera(a=(0.0, 30.0, 2.0)), 20, 20, tf, shader="Volume",
                              sample_rate=0.5, density=0.3)
            finally:
                b.close()
    finally:
        c.close()


def test_captured_render_follows_the_knots(ctx):
    """A render captured by the caller replays with the knots of that time."""
    torch = pytest.importorskip("torch")
    c = Case(ctx, voxels("u8", (64, 64, 64)), 32, 1, tf=knots("first"))
    out = torch.zeros(48 * 40 * 4, dtype=torch.uint8, device="cuda")
    p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3)
    view = hy.camera_view(c.vol, camera())
    try:
        s = torch.cuda.ExternalStream(ctx.stream)
        hy.render(ctx, c.vol, p, view, 48, 40)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            hy.render_device(ctx, c.vol, p, view, 48, 40, out.data_ptr())
        for tf in ("ends", "inside", "first"):
            ctx.set_transfer_fn(knots(tf))
            want = hy.render(ctx, c.vol, p, view, 48, 40).rgba
            out.zero_()
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy().reshape(40, 48, 4), want), tf
        del g
    finally:
        c.close()


@pytest.mark.parametrize("density", [0.0, 1e-3, 0.05, 0.7, 3.0, -0.4])
@pytest.mark.parametrize("composite", [False, True])
def test_blocks(ctx, density, composite):
    """The Blocks march takes a brick's steps in runs: opacities that pass the
    threshold early, late and never, fall, or leave [0, 1]; rays along the axes;
    bricks of fewer and of more steps than a run."""
    for bs, rate in ((8, 0.25), (32, 1.0), (24, 2.0)):
        c = Case(ctx, voxels("u8", (64, 48, 50)), bs, 1)
        try:
            for cam in (camera(), camera("ptu", a=(0.0, 0.0, 2.2)),
                        camera("ptu", a=(0.1, 0.2, 0.05), target=(1.0, 0.3, 0.2))):
                check(c, cam, 61, 47, f"{density} bs{bs}", shader="Blocks", mode="Volume",
                      density=density, sample_rate=rate, composite=composite)
                check(c, cam, 33, 35, f"solid bs{bs}", shader="Blocks", mode="Solid",
                      density=density, sample_rate=rate, composite=composite)
        finally:
            c.close()


@pytest.mark.parametrize("shader,mode", [("Volume", "Default"), ("Volume", "Partition"),
                                         ("Isosurface", "Position"), ("Blocks", "Volume"),
                                         ("Blocks", "Solid")])
@pytest.mark.parametrize("dtype,pad", [("u8", 1), ("u8", 0), ("f32", 1)])
def test_films(ctx, shader, mode, dtype, pad):
    """The emit pass leaves the plain march's film, byte for byte, in each form
    (sizes on both sides of 155,648 and 466,944 rays), and a march pass leaves
    the film of rays that have marched to their end."""
    torch = pytest.importorskip("torch")
    c = Case(ctx, voxels(dtype, (70, 61, 52)), 32, pad, tf=knots("ends"))
    try:
        fb = 48 if shader == "Blocks" else 64
        for W, H in ((41, 33), (395, 393), (397, 394), (690, 680)):
            cam = camera(a=(-50.0, 20.0, 1.9))
            p = hy.shader_params(shader=shader, mode=mode, sample_rate=0.5, density=0.3, rank=0.4)
            if shader == "Isosurface":
                hy.iso_lighting(c.vol, cam, p)
            view = hy.camera_view(c.vol, cam)
            film = torch.zeros(H * W * fb, dtype=torch.uint8, device="cuda")
            hy.shade_pass(ctx, c.vol, p, hy._abi.PASS_RAY_EMIT, view, film.data_ptr(), W, H)
            ctx.synchronize()
            ref = orc.render(c.ov, c.tf, orc.params_from(p), view_array(view), W, H, want_film=True)
            got = film.cpu().numpy().reshape(H, W, fb)
            assert np.array_equal(got, ref["film"]), (shader, mode, W, H)
        before = film.clone()
        hy.shade_pass(ctx, c.vol, p, hy._abi.PASS_RAY_MARCH, None, film.data_ptr(), W, H)
        ctx.synchronize()
        assert torch.equal(before, film)
    finally:
        c.close()
