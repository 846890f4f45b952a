"""The adjoint through range profiles after a focus: it may read the focus's table, and must not
depend on how that focus was planned."""
import numpy as np
import pytest

from sarlabtdc import scenes

pytestmark = pytest.mark.gpu

INF = float("inf")


def _processor(band, height=0.05, n_pri=520, nx=57, ny=131, n_samples=192):
    import _sarlabtdc

    sc = scenes.small_scene(seed=41, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=1e-3, rail_len=0.52,
                            jitter=0.2e-3, height=height, y0=0.02, device="cuda")
    api = sc.api_arrays()
    api["velocity"][..., 0] = 0.08
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setChirpPositionsF64(sc.positions)
    p.setFocusGridF64(sc.grid)
    p.prepare(0.0, band, False, False, True)
    p.uploadGrid()
    return p


def _gradient(p, n, seed=2):
    import torch

    rng = np.random.default_rng(seed)
    g = (rng.normal(size=p.numPixels()) + 1j * rng.normal(size=p.numPixels())).astype(np.complex64)
    return torch.from_numpy(g).cuda(), torch.empty((n, 3), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("band", [INF, 14.0])
def test_adjoint_after_anchored_ranges_were_switched(cuda_device, band):
    """A focus with every pixel's own range, then anchors on: the adjoint of groups of 8 is the one
    without a focus before it, bit for bit; and the other way round."""
    import torch

    p = _processor(band)
    g, grad = _gradient(p, 520)
    img = torch.empty(p.numPixels(), dtype=torch.complex64, device="cuda")
    for before, after in ((False, True), (True, False)):
        alone = _processor(band)
        alone.setAnchoredRanges(after)
        alone.adjointDevice(g, grad)
        ref = grad.cpu().numpy()
        p.setAnchoredRanges(before)
        p.focusDevice(img)
        p.check()
        st = p.lastStats()
        assert st["stage_samples"] == 0 and st["anchor_pixels"] == (8 if before else 0)
        p.setAnchoredRanges(after)
        p.adjointDevice(g, grad)
        assert np.any(ref)
        np.testing.assert_array_equal(grad.cpu().numpy(), ref)
