"""The differentiable renderer at the sizes where its kernels change form: odd
and even padded edges and more than one column of slices in the gather texture,
segments that are no multiple of the samples in flight, one knot, values out of
[0, 1], and launches on both sides of 8 warps of rays a scheduler (155,648
rays on 152 SMs).  The forward is the oracle's float forward; the gradients
face the oracle's FP64 ones with the 1e-3 of the repository's other gradient
tests (volumes end in an empty rim below 1, away from the float forward's own
discontinuities)."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from hydrant_gb300 import fit
from oracle import oracle as orc
from tests._harness import view_array

pytestmark = pytest.mark.gpu


def inputs(ctx, n, nviews, ntf):
    vol = np.zeros((n, n, n), np.float32)
    vol[2:-2, 2:-2, 2:-2] = hy.synth_blobs_f32(4, (n - 4,) * 3, 6) * np.float32(0.9)
    holder = hy.Volume(ctx, np.ones((8, 8, 8), np.float32), 8, 1)
    views = fit.orbit_views(holder, 7, nviews)
    holder.close()
    tf = np.clip(fit.seeded_tf(9, ntf) * 0.8 + 0.1, 0, 1).astype(np.float32)
    return vol, tf, views, np.stack([view_array(v) for v in views])


@pytest.mark.parametrize("n,nviews,W,H,ntf,k,rate", [
    (23, 2, 17, 13, 5, 1, 1.0), (24, 2, 33, 7, 16, 3, 1.0), (9, 3, 20, 20, 1, 64, 2.0),
    (200, 1, 24, 19, 33, 32, 0.5), (24, 1, 395, 394, 16, 7, 0.5), (24, 1, 395, 395, 256, 32, 0.5)])
def test_forward_and_gradients(ctx, n, nviews, W, H, ntf, k, rate):
    torch = pytest.importorskip("torch")
    vol, tf, views, va = inputs(ctx, n, nviews, ntf)
    r = fit.DiffRenderer(ctx, n, views, W, H, ntf, sample_rate=rate, density=0.7, ckpt_k=k)
    tv, tt = torch.from_numpy(vol).cuda(), torch.from_numpy(tf).cuda()
    img = r.forward(tv, tt)
    plain = r.forward(tv, tt, keep=False)
    torch.cuda.synchronize()
    ref = orc.diff_forward(vol, tf, va, W, H, sample_rate=rate, density=0.7)
    assert np.array_equal(img.cpu().numpy(), ref) and torch.equal(img, plain)
    target = np.zeros_like(ref, dtype=np.float64)
    _, img64, dv64, dt64 = orc.diff_loss_grad64(vol, tf, va, W, H, target, sample_rate=rate,
                                                density=0.7)
    img = r.forward(tv, tt)
    dv, dt = r.backward(tv, tt, (2.0 * img).contiguous())
    torch.cuda.synchronize()
    dv, dt = dv.cpu().numpy().astype(np.float64), dt.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(dt - dt64) <= 1e-3 * np.linalg.norm(dt64)
    if ntf > 1:  # one knot: the image does not depend on the voxels
        assert np.linalg.norm(dv - dv64) <= 1e-3 * np.linalg.norm(dv64)
    else:
        assert not dv.any() and not dv64.any()


def test_values_out_of_range(ctx):
    """Below 0, above 1, infinite and NaN voxels: transparent, as in the oracle."""
    torch = pytest.importorskip("torch")
    vol, tf, views, va = inputs(ctx, 24, 2, 16)
    vol[5:9] -= 0.6
    vol[12:15] += 0.7
    vol[16, 3:9, 4:7] = np.inf
    vol[18, 3:9, 4:7] = np.nan
    r = fit.DiffRenderer(ctx, 24, views, 31, 29, 16, ckpt_k=5)
    img = r.forward(torch.from_numpy(vol).cuda(), torch.from_numpy(tf).cuda())
    torch.cuda.synchronize()
    ref = orc.diff_forward(vol, tf, va, 31, 29)
    assert np.array_equal(img.cpu().numpy(), ref, equal_nan=True)
