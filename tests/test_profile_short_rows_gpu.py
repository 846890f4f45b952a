"""Which kernel focuses short rows: with every pixel its own range (shuffled pixels), range profiles from
17 samples on, 33 under a finite band; with shared anchors at any length. Against the FP64 oracle,
2e-4 under the band (chirps at its edge), else 3e-6 for profiles and 1e-5 for the direct kernel (its
error grows as the rows get fewer samples to average over)."""
import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import problem_from_api, rel_l2

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("n_samples,band,shuffled,profiles", [
    (16, INF, True, False), (17, INF, True, True), (16, INF, False, True),
    (32, 10.0, True, False), (33, 10.0, True, True), (32, 10.0, False, True),
])
def test_short_rows(cuda_device, n_samples, band, shuffled, profiles):
    import _sarlabtdc

    nx, ny = 160, 150
    n_pri = int(5.2e8 / (nx * ny * n_samples))
    sc = scenes.small_scene(seed=n_samples, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=0.2e-3, rail_len=0.6,
                            device="cuda")
    api = sc.api_arrays()
    api["velocity"][..., 0] = 0.08
    grid = sc.grid.astype(np.float32)
    if shuffled:
        grid = grid.reshape(-1, 3)[np.random.default_rng(1).permutation(nx * ny)].reshape(ny, nx, 3)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.start(0.0, band, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert (st["stage_samples"] == 0) == profiles
    pix = np.random.default_rng(2).choice(img.size, 60, replace=False)
    ref = oracle.focus(problem_from_api(api, grid), oracle.Opts(applyRangeWin=False, dopplerBandwidth=band), pixels=pix)
    assert rel_l2(img[pix], ref) <= (2e-4 if np.isfinite(band) else 3e-6 if profiles else 1e-5)
