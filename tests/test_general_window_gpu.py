"""GPU parity of the FP32 general kernels (csrc/tdc_general.cu) where per-sample windows leave most
chirps out of band: a warp leaves out a chirp only where no sample of it can be in band.

Tolerance 2e-4, as for every finite band: a sample at the inclusive edge may fall on either side
in FP32 and FP64."""
import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import rel_l2

pytestmark = pytest.mark.gpu


def _scene(nx, ny, n_pri, n_samples, moving, uneven, spread):
    sc = scenes.small_scene(seed=nx + n_samples, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=2e-3,
                            rail_len=0.8, device="cuda")
    api = sc.api_arrays()
    rng = np.random.default_rng(9)
    u = np.arange(n_samples) / n_samples
    vel = np.zeros_like(api["velocity"])
    vel[..., 0] = 0.08 * (1.0 + spread * np.sin(2 * np.pi * u)[None, :])
    vel[..., 1] = 0.02 * rng.normal(size=(n_pri, 1))
    api["velocity"] = vel.astype(np.float32)
    if moving:
        pos = api["position"].astype(np.float64)
        pos = pos + 1e-4 * np.sin(2 * np.pi * 3 * u[None, :, None] + rng.uniform(0, 6.28, (n_pri, 1, 1)))
        api["position"] = pos.astype(np.float32)
    if uneven:
        t = api["sampleTimes"].astype(np.float64)
        api["sampleTimes"] = (t + 0.2 * (t[1] - t[0]) * np.sin(0.1 * np.arange(n_samples))).astype(np.float32)
    return sc, api


@pytest.mark.parametrize("moving,uneven", [(True, False), (False, False), (False, True), (True, True)])
@pytest.mark.parametrize("nx,ny,n_pri,n_samples,centre,band,spread", [
    (33, 40, 150, 100, 0.0, 8.0, 0.02),
    (64, 64, 129, 75, 3.0, 12.0, 0.3),    # windows that sweep through the band within a chirp
    (40, 33, 40, 5000, 0.0, 8.0, 0.02),   # rows staged in segments
])
def test_window_skips_only_dead_chirps(cuda_device, nx, ny, n_pri, n_samples, centre, band, spread, moving, uneven):
    import _sarlabtdc

    sc, api = _scene(nx, ny, n_pri, n_samples, moving, uneven, spread)
    grid = sc.grid.astype(np.float32)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.start(centre, band, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert st["path_name"] == "general" and st["general_variant"] == 2 + moving + 4 * uneven
    pix = np.unique(np.concatenate([[0, nx - 1, nx, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 60, replace=False)]))
    prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=api["position"],
                          velocity=api["velocity"], attitude=api["attitude"], modRate=api["modRate"],
                          startFreq=api["startFreq"], grid=grid)
    ref = oracle.focus(prob, oracle.Opts(dopplerWinCenter=centre, dopplerBandwidth=band, applyRangeWin=False),
                       pixels=pix)
    assert rel_l2(img[pix], ref) <= 2e-4


def test_non_finite_sample_is_not_skipped(cuda_device):
    """A sample that is not a number reaches every pixel whose chunk is kept, in band or not."""
    import _sarlabtdc

    sc, api = _scene(64, 64, 100, 100, True, False, 0.02)
    raw = api["rawData"].copy()
    raw[0, 7] = np.nan + 0j
    api["rawData"] = raw
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(sc.grid.astype(np.float32))
    p.setSkipTest(False)
    p.start(0.0, 3.0, False, False, True)
    assert np.all(np.isnan(p.getFocusedImage()))
