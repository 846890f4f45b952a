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


def test_adjoint_beside_a_focus_on_another_stream(cuda_device):
    """A focus in flight on one stream, the adjoint enqueued on another with no order between them:
    both give what they give alone, bit for bit; with the table of the focus, and with another
    (anchored ranges switched in between)."""
    import torch

    kw = dict(height=0.3, n_pri=1500, nx=800, ny=600, n_samples=256)
    p = _processor(INF, **kw)
    g, grad = _gradient(p, 1500)
    img, ref_img = (torch.empty(p.numPixels(), dtype=torch.complex64, device="cuda") for _ in range(2))
    refs = {}
    for anchored in (True, False):
        alone = _processor(INF, **kw)
        alone.setAnchoredRanges(anchored)
        alone.adjointDevice(g, grad)
        refs[anchored] = grad.cpu().numpy()
        if anchored:
            alone.focusDevice(ref_img)
            alone.check()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for anchored in (True, False):
        p.setAnchoredRanges(True)
        with torch.cuda.stream(one):
            p.focusDevice(img)
        p.setAnchoredRanges(anchored)
        with torch.cuda.stream(two):
            p.adjointDevice(g, grad)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(grad.cpu().numpy(), refs[anchored])
        np.testing.assert_array_equal(img.cpu().numpy(), ref_img.cpu().numpy())
