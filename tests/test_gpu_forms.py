"""The marches' forms that the other tests do not reach, against the oracle:
images, floats and sample counts equal, bit for bit."""

import numpy as np
import pytest

from tests._harness import Case, camera
from tests.test_gpu_skip import check, voxels

pytestmark = pytest.mark.gpu


def dense_knots():
    k = np.random.default_rng(7).uniform(0.1, 1.0, (9, 4)).astype(np.float32)
    return k


@pytest.mark.parametrize("wh", [(311, 312), (313, 311), (394, 395), (395, 395), (684, 682), (684, 683)])
@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_no_free_cells(ctx, wh, dtype):
    """Knots without a transparent run: samples in flight up to 5, 8 and 24 warps
    of rays a scheduler (97,280, 155,648 and 466,944 rays on 152 SMs) by gathers,
    loads and f32 loads."""
    c = Case(ctx, voxels(dtype, (70, 61, 52)), 32, 1, tf=dense_knots())
    try:
        for density in (0.01, 0.3):
            check(c, camera(), *wh, f"{wh} {dtype} {density}", shader="Volume", sample_rate=0.5,
                  density=density)
    finally:
        c.close()
