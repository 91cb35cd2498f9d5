"""The marches' forms that the other tests do not reach, against the oracle:
images, floats and sample counts equal, bit for bit."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from hydrant_gb300 import _abi
from oracle import oracle as orc
from tests._harness import Case, camera, view_array
from tests.test_gpu_skip import check, knots, voxels

pytestmark = pytest.mark.gpu


def dense_knots():
    k = np.random.default_rng(7).uniform(0.1, 1.0, (9, 4)).astype(np.float32)
    return k


@pytest.mark.parametrize("wh", [(278, 279), (279, 280), (311, 312), (313, 311), (394, 395), (395, 395), (684, 682), (684, 683)])
@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_no_free_cells(ctx, wh, dtype):
    """Knots without a transparent run: samples in flight up to 4, 5, 8 and 24 warps
    of rays a scheduler (77,824, 97,280, 155,648 and 466,944 rays on 152 SMs) by
    gathers, loads and f32 loads."""
    c = Case(ctx, voxels(dtype, (70, 61, 52)), 32, 1, tf=dense_knots())
    try:
        for density in (0.01, 0.3):
            check(c, camera(), *wh, f"{wh} {dtype} {density}", shader="Volume", sample_rate=0.5,
                  density=density)
    finally:
        c.close()


@pytest.mark.parametrize("wh", [(341, 342), (342, 342), (395, 396)])
@pytest.mark.parametrize("dtype,bs", [("u8", 16), ("u8", 32), ("f32", 16), ("f32", 32)])
def test_lines_between_the_forms(ctx, wh, dtype, bs):
    """Isosurfaces on both sides of 6 warps of rays a scheduler (116,736 rays), and
    dense knots in bricks below and from 32 voxels on, per view and batched."""
    c = Case(ctx, voxels(dtype, (70, 61, 52)), bs, 1, tf=dense_knots())
    W, H = wh
    try:
        check(c, camera(), W, H, f"{wh} {dtype} {bs} iso", shader="Isosurface", mode="Position",
              sample_rate=0.5, isovalue=0.4)
        check(c, camera(), W, H, f"{wh} {dtype} {bs}", shader="Volume", sample_rate=0.5, density=0.2)
        p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.2)
        view = hy.camera_view(c.vol, camera())
        for sizes in ([(W, H)], [(W, H // 2), (W, H // 4)]):
            b = hy.Batch(ctx, c.vol, p, [(view, w, h) for w, h in sizes])
            try:
                for img, (w, h) in zip(b.render(), sizes):
                    r = orc.render(c.ov, c.tf, orc.params_from(p), view_array(view), w, h)
                    assert np.array_equal(img, r["rgba"]), (w, h)
            finally:
                b.close()
    finally:
        c.close()


@pytest.mark.parametrize("bs", [64, 128])
@pytest.mark.parametrize("wh", [(31, 27), (197, 200), (396, 395), (690, 684)])
def test_compile_time_edges(ctx, bs, wh):
    """Bricks of 64^3 and 128^3 voxels with an apron (compile-time edges of 66 and
    130): every form of the Volume and Isosurface march, in one march, composited
    and over films."""
    torch = pytest.importorskip("torch")
    dims = (150, 140, 133)
    c = Case(ctx, voxels("u8", dims), bs, 1, tf=knots("ends"))
    W, H = wh
    try:
        for composite in (False, True):
            check(c, camera(a=(-50.0, 20.0, 1.9)), W, H, f"{bs} {wh} {composite}", shader="Volume",
                  sample_rate=0.25, density=0.2, composite=composite)
            check(c, camera(a=(-50.0, 20.0, 1.9)), W, H, f"{bs} {wh} {composite} iso",
                  shader="Isosurface", mode="Position", sample_rate=0.25, isovalue=0.4,
                  composite=composite)
        for shader, mode in (("Volume", "Default"), ("Isosurface", "Position")):
            for gather in (True, False):
                c.vol.set_gather_sampling(gather)
                cam = camera(a=(-50.0, 20.0, 1.9))
                p = hy.shader_params(shader=shader, mode=mode, sample_rate=0.25, density=0.2,
                                     isovalue=0.4)
                if shader == "Isosurface":
                    hy.iso_lighting(c.vol, cam, p)
                view = hy.camera_view(c.vol, cam)
                # the emit pass in one go, and cut short with march passes after it
                ref = orc.render(c.ov, c.tf, orc.params_from(p), view_array(view), W, H,
                                 want_film=True)["film"]
                film = torch.zeros(H * W * 64, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
                hy.shade_pass(ctx, c.vol, p, hy._abi.PASS_RAY_EMIT, view, film.data_ptr(), W, H)
                ctx.synchronize()
                assert np.array_equal(film.cpu().numpy().reshape(H, W, 64), ref), (shader, gather)
                p.max_steps = 60
                part = orc.render(c.ov, c.tf, orc.params_from(p), view_array(view), W, H,
                                  want_film=True)["film"].copy()
                part.view(np.int32)[..., 6][part.view(np.int32)[..., 6] == 0] = 40
                dev = torch.from_numpy(part.copy()).cuda()
                torch.cuda.synchronize()
                hy.shade_pass(ctx, c.vol, p, hy._abi.PASS_RAY_MARCH, None, dev.data_ptr(), W, H)
                ctx.synchronize()
                orc.march_film(c.ov, c.tf, orc.params_from(p), part, W, H, nthreads=8)
                assert np.array_equal(dev.cpu().numpy(), part), (shader, gather)
    finally:
        c.vol.set_gather_sampling(True)
        c.close()


@pytest.mark.parametrize("bs", [16, 64, 128])
@pytest.mark.parametrize("gather", [True, False])
def test_batch_by_the_rule(ctx, bs, gather):
    """Batches whose samples in flight the library chooses (steps_per_iter 0), below
    and above 8 warps of rays a scheduler, with and without free cells, composited
    too, view by view against the oracle."""
    c = Case(ctx, voxels("u8", (150, 140, 133)), bs, 1)
    c.vol.set_gather_sampling(gather)
    try:
        for name, tf in (("ends", knots("ends")), ("dense", dense_knots())):
            ctx.set_transfer_fn(tf)
            for sizes in (((60, 50), (33, 71)), ((410, 400), (64, 64))):
                for composite in (False, True):
                    p = hy.shader_params(shader="Volume", sample_rate=0.25, density=0.2,
                                         composite=composite)
                    views = [(hy.camera_view(c.vol, camera(a=(20.0 * i, 30.0, 2.0))), W, H)
                             for i, (W, H) in enumerate(sizes)]
                    b = hy.Batch(ctx, c.vol, p, views)
                    try:
                        assert b.config.steps_per_iter == 0
                        b.set_counting(True)
                        got, n, want = b.render(), ctx.stats().samples, 0
                        for img, (view, W, H) in zip(got, views):
                            r = orc.render(c.ov, tf, orc.params_from(p), view_array(view), W, H)
                            want += r["samples"]
                            assert np.array_equal(img, r["rgba"]), (name, W, H, composite)
                        assert n == want, (name, sizes, composite)
                    finally:
                        b.close()
    finally:
        c.vol.set_gather_sampling(True)
        c.close()


@pytest.mark.parametrize("sampler", [_abi.PAGER_LOADS, _abi.PAGER_GATHERS])
@pytest.mark.parametrize("level", [0, 2])
def test_paged_with_few_free_cells(ctx, sampler, level):
    """Realtime frames whose knots are transparent where hardly a cell lies (no grid
    by the coarse stand-ins' count; without a coarse level always one), then where
    most lie, then nowhere."""
    torch = pytest.importorskip("torch")
    vox = np.maximum(voxels("u8", (96, 64, 80)), 1)
    vol, ov = hy.Volume(ctx, vox, 16, 1), orc.OracleVolume(vox, 16, 1)
    store = hy.Store.from_volume(vol)
    if level:
        store.build_coarse(level)
        ov.build_coarse(level)
    pg = hy.Pager(ctx, store, max(4, vol.info.nonempty // 3), _abi.PAGER_REALTIME, sampler=sampler)
    few = dense_knots()
    few[7:, 3] = 0
    try:
        for f, tf in enumerate((few, knots("first"), dense_knots())):
            cam = hy.camera_orbit((25.0 + 40.0 * f, 30.0, 1.4))
            for W, H in ((57, 43), (317, 315), (397, 394)):
                ctx.set_transfer_fn(tf)
                p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3,
                                     count_samples=True)
                out = torch.zeros(W * H * 4, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
                pg.render(p, cam, W, H, out.data_ptr())
                samples = ctx.stats().samples
                ov.set_present(pg.present())
                op = orc.params_from(p)
                op.lowest_blkcnt = ov.lowest_blkcnt if level else 0
                ref = orc.render(ov, tf, op, view_array(hy.camera_view(pg.volume, cam)), W, H)
                assert np.array_equal(out.cpu().numpy().reshape(H, W, 4), ref["rgba"]), (f, W)
                assert samples == ref["samples"], (f, W)
    finally:
        pg.close()
        store.close()
        vol.close()
