"""The partial-sum reductions (csrc/tdc_focus.cu) where nearly everything cancels: every chirp but one
has an opposite at the same position, 1e9 times the one that is left. Few enough chirps and tiles
that every chirp is a group of its own, so the opposites' partial sums are equal bit for bit, and
the image is that of the one chirp by the same plan.

Tolerance: 2e-7 of the image, one rounding to FP32 beside the n^2 2^-74 of the largest partial sum
that the sums keep to (1e-8 of what is left). FP64 leaves n 2^-53 of it, up to 1e-4 and 4e-6 as a rule."""
import numpy as np
import pytest

from sarlabtdc import scenes
from tdc_testutil import rel_l2, run_engine

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("nx,ny,half", [(8, 8, 200), (33, 1, 100), (40, 12, 6), (31, 1, 7),
                                        (128, 66, 150),    # eight slices
                                        (210, 195, 30)])   # many pixels: a thread each
def test_opposite_chirps_cancel(cuda_device, nx, ny, half):
    n_pri = 2 * half + 1
    sc = scenes.small_scene(seed=nx + half, n_pri=n_pri, n_samples=64, nx=nx, ny=ny, device="cuda")
    api = sc.api_arrays()
    raw, pos = api["rawData"].copy(), np.array(api["position"])
    rng = np.random.default_rng(3)
    raw[:half] *= (1e9 * rng.uniform(0.3, 1.0, (half, 1))).astype(np.float32)
    order = rng.permutation(half)
    raw[half + 1 :] = -raw[:half][order]
    pos[half + 1 :] = pos[:half][order]
    alone = raw * (np.arange(n_pri) == half)[:, None].astype(np.float32)
    args = (0.0, INF, False, False, True)
    img, _, _ = run_engine(dict(api, rawData=raw, position=pos), sc.grid, args)
    ref, _, _ = run_engine(dict(api, rawData=alone, position=pos), sc.grid, args)
    assert np.abs(ref).max() > 0
    err = rel_l2(img, ref)
    assert err <= 2e-7, err
