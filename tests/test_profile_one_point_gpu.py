"""GPU behaviour of the focus through range profiles (csrc/tdc_profile.cu) where a group's pixels are
one point: its reach is zero, and ranges down to zero are not below it."""
import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import problem_from_api, rel_l2

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("times,n_pri,group,band", [(8, 300, 8, INF), (16, 800, 16, INF), (8, 300, 8, 500.0)])
def test_antenna_on_a_group_of_one_point(cuda_device, times, n_pri, group, band):
    """Every grid point `times` times in a row, the antenna on one of them for one chirp: its window is
    zero there. 4e-6 relative L2 against the FP64 oracle, as for runs along an axis (under the band,
    2e-4: a chirp at its edge)."""
    import _sarlabtdc

    sc = scenes.small_scene(seed=8, n_pri=n_pri, n_samples=160, nx=64, ny=1280 // times * 8, spacing=2e-3, height=0.05,
                            y0=0.01, device="cuda")
    api = sc.api_arrays()
    api["velocity"][..., 0] = 0.08
    grid = np.repeat(sc.grid.reshape(-1, 3)[: 81920 // times].astype(np.float32), times, axis=0)[None]
    pos = np.array(api["position"])
    pos[150, :, :] = grid[0, 40 * times]
    api["position"] = pos
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.setSkipTest(False)
    p.start(0.0, band, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert st["stage_samples"] == 0 and st["anchor_pixels"] == group
    pix = np.arange(38 * times, 44 * times, 3)
    ref = oracle.focus(problem_from_api(api, grid), oracle.Opts(applyRangeWin=False, dopplerBandwidth=band,
                                                                skip_test=False), pixels=pix)
    assert np.all(np.isfinite(img)) and np.any(ref)
    assert rel_l2(img[pix], ref) <= (4e-6 if np.isinf(band) else 2e-4)
