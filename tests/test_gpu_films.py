"""A march pass over films that the caller wrote: rays whose opacity, step size
and theta / phi no march of this library leaves together take every sample, as in
the oracle, whatever the skip grid says."""

import numpy as np
import pytest

import hydrant_gb300 as hy
from oracle import oracle as orc
from tests._harness import Case
from tests.test_gpu_skip import knots, voxels

pytestmark = pytest.mark.gpu


def film(W, H, dims):
    """Rays from the z = 0 face into the volume, a state per column."""
    rng = np.random.default_rng(3)
    f = np.zeros((H, W, 16), np.float32)
    f[..., 0] = rng.uniform(0.1, 0.9, (H, W)) * dims[0]
    f[..., 1] = rng.uniform(0.1, 0.9, (H, W)) * dims[1]
    f[..., 2] = 0.01
    d = rng.uniform(-0.4, 0.4, (H, W, 3)) + (0.0, 0.0, 1.0)
    f[..., 3:6] = d / np.linalg.norm(d, axis=-1, keepdims=True)
    f[..., 6].view(np.int32)[:] = 90
    f[..., 12:16] = (0.0, 0.0, 0.0, 1.0)
    inf, nan = np.inf, np.nan
    states = [(0.0, 1, 1.0), (0.5, 1, 0.4), (0.9, 1, 1.0), (0.9, 4, 1.0), (0.86, 16, 1.0),
              (0.95, 1, 0.2), (0.95, 4, 1.0), (0.95, 16, 1.0), (1.2, 16, 1.0), (1.2, 2, 1.0),
              (-0.3, 1, 1.0), (0.3, 3, 1.0), (inf, 16, 1.0), (nan, 1, 1.0), (0.2, 1, inf),
              (0.2, 1, nan)]
    for x in range(W):
        vw, ss, phi = states[x % len(states)]
        f[:, x, 7].view(np.int32)[:] = ss
        f[:, x, 8:11] = 0.1
        f[:, x, 11] = vw
        f[:, x, 15] = phi
    return f


@pytest.mark.parametrize("dtype,pad", [("u8", 1), ("f32", 1), ("u8", 0)])
@pytest.mark.parametrize("wh", [(48, 21), (400, 395)])
def test_written_films(ctx, dtype, pad, wh):
    torch = pytest.importorskip("torch")
    W, H = wh
    tf = knots("ends")
    c = Case(ctx, voxels(dtype, (70, 61, 52)), 16, pad, tf=tf)
    try:
        dims = [d / 16.0 for d in (70, 61, 52)]
        p = hy.shader_params(shader="Volume", sample_rate=0.5, density=0.3, count_samples=True)
        want = film(W, H, dims)
        dev = torch.from_numpy(want.copy()).cuda()
        torch.cuda.synchronize()
        hy.shade_pass(ctx, c.vol, p, hy._abi.PASS_RAY_MARCH, None, dev.data_ptr(), W, H)
        samples = ctx.stats().samples
        ref = want.view(np.uint8).reshape(H, W, 64).copy()
        n = orc.march_film(c.ov, tf, orc.params_from(p), ref, W, H, nthreads=8)
        got, ref = dev.cpu().numpy(), ref.view(np.float32).reshape(H, W, 16)
        assert np.array_equal(got[..., 6:8].view(np.int32), ref[..., 6:8].view(np.int32))
        got[..., 6:8] = ref[..., 6:8] = 0
        assert np.array_equal(got, ref, equal_nan=True)
        assert samples == n
    finally:
        c.close()
