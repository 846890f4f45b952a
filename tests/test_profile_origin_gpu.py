"""GPU parity of the focus through range profiles with FP64 positions and grids far from the
origin, where the high floats of the double-float pairs alone are off by as much as the ranges
can be resolved: the same scenes as at the origin, all of it moved.

Tolerances: the 3e-6 of the focus through range profiles (4e-6 on runs along an axis, phases
unreduced), relative L2 against the FP64 oracle, and what a pair of floats holds of the moved
coordinates, 2^-49 of them rms on each axis of antenna and pixel: 2 x 2 pi 525 cycles / m x that x
sqrt(3), below 1e-8 at 1 km."""
import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import rel_l2

pytestmark = pytest.mark.gpu

INF = float("inf")
KM = np.array([1234.56789, -987.654321, 111.1111])


def _moved(shift, **kw):
    sc = scenes.small_scene(device="cuda", jitter=0.3e-3, **kw)
    sc.positions = sc.positions + shift
    sc.grid = sc.grid + shift
    return sc


def _processor(sc, api=None, anchored=True, band=INF):
    import _sarlabtdc

    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*(sc.api_arrays() if api is None else api).values())
    p.setChirpPositionsF64(sc.positions)
    p.setFocusGridF64(sc.grid)
    p.setAnchoredRanges(anchored)
    p.prepare(0.0, band, False, False, True)
    p.uploadGrid()
    return p


def _problem(sc, api):
    return oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=sc.positions,
                          velocity=api["velocity"][:, 0, :], modRate=api["modRate"], startFreq=api["startFreq"],
                          grid=sc.grid)


def _focus(p):
    import torch

    img = torch.empty(p.numPixels(), dtype=torch.complex64, device="cuda")
    p.focusDevice(img)
    p.check()
    st = p.lastStats()
    assert st["path_name"] == "fp32_bulk" and st["stage_samples"] == 0
    return img.cpu().numpy(), st["anchor_pixels"]


@pytest.mark.parametrize("nx,ny,n_pri,n_samples,spacing,height,group", [
    (133, 202, 300, 160, 1e-3, 0.1, 8),
    (256, 320, 800, 160, 1e-3, 0.3, 16),
    (77, 154, 169, 300, 8e-3, 0.05, 2),
    (57, 131, 300, 256, 1e-3, 0.02, 8),   # ranges too short for the series
])
def test_far_grid_focus(cuda_device, nx, ny, n_pri, n_samples, spacing, height, group):
    sc = _moved(KM, seed=nx, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing, height=height)
    img, anchor = _focus(_processor(sc))
    assert anchor == group
    pix = np.unique(np.concatenate([[0, nx - 1, nx, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 60, replace=False)]))
    ref = oracle.focus(_problem(sc, sc.api_arrays()), oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    assert np.all(np.isfinite(img))
    err = rel_l2(img[pix], ref)
    assert err <= 4e-6, err


@pytest.mark.parametrize("anchored", [True, False])
def test_far_grid_adjoint(cuda_device, anchored):
    """An image gradient on a few pixels only, so that the oracle need not take the others."""
    import torch

    sc = _moved(KM, seed=63, n_pri=300, n_samples=192, nx=83, ny=119, spacing=2e-3)
    p = _processor(sc, anchored=anchored)
    n = p.numPixels()
    rng = np.random.default_rng(4)
    pix = np.sort(rng.choice(n, 400, replace=False))
    g = np.zeros(n, np.complex64)
    g[pix] = (rng.normal(size=pix.size) + 1j * rng.normal(size=pix.size)).astype(np.complex64)
    grad = torch.empty((sc.n_pri, 3), dtype=torch.float64, device="cuda")
    p.adjointDevice(torch.from_numpy(g).cuda(), grad)
    ref = oracle.adjoint_offsets(_problem(sc, sc.api_arrays()), oracle.Opts(applyRangeWin=False), None,
                                 g[pix].astype(np.complex128), pixels=pix)
    err = rel_l2(grad.cpu().numpy(), ref)
    assert err <= 4e-6, err


def test_antenna_on_a_far_pixel(cuda_device):
    """For one chirp the antenna is on a pixel that is not its group's anchor: the pixel's window is
    zero there (a Doppler frequency that is not a number), the others' is not."""
    sc = _moved(KM, seed=8, n_pri=300, n_samples=256, nx=72, ny=110, height=0.02, y0=0.01)
    sc.positions[150] = sc.grid[40, 21]
    img, anchor = _focus(_processor(sc))
    assert anchor == 8
    pix = np.arange(40 * 72 + 16, 40 * 72 + 32)
    ref = oracle.focus(_problem(sc, sc.api_arrays()), oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    err = rel_l2(img[pix], ref)
    assert err <= 4e-6, err


# Map coordinates. A pair of floats holds them to 2^-29 m at 1e6 m and 2^-26 m at 4.5e6 m (ulp of the low
# float), and differences of low floats are rounded to the same, once for antenna - anchor and once for
# pixel - anchor: 3400 rad / m x ulp x (sqrt(2 / 12) + 2 x 2 / sqrt(12)) = 1.0e-5 and 8e-5 rad rms,
# relative L2 beside the 4e-6.
FAR = [(np.array([1.0e6, -0.7e6, 0.1e6]) + 0.123, 1.4e-5), (np.array([4.5e6, 3.3e6, -1.0e6]) + 0.456, 8.4e-5)]


@pytest.mark.parametrize("shift,tol", FAR)
@pytest.mark.parametrize("nx,ny,n_pri,n_samples,spacing,height,anchored", [
    (133, 202, 300, 160, 1e-3, 0.3, True),
    (256, 320, 800, 160, 1e-3, 0.3, True),
    (256, 64, 400, 256, 0.3e-3, 0.3, True),   # a grid narrower than half an ulp of its coordinates
    (77, 154, 169, 300, 8e-3, 0.3, True),
    (100, 120, 300, 160, 1e-3, 0.3, False),
])
def test_map_coordinates_focus(cuda_device, nx, ny, n_pri, n_samples, spacing, height, anchored, shift, tol):
    """The table's place and extent, and the groups' reach, follow the low parts of the grid too."""
    sc = _moved(shift, seed=nx, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing, height=height)
    img, anchor = _focus(_processor(sc, anchored=anchored))
    at_origin = _moved(0.0, seed=nx, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing, height=height)
    assert anchor == _focus(_processor(at_origin, anchored=anchored))[1]
    pix = np.unique(np.concatenate([[0, nx - 1, nx, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 60, replace=False)]))
    ref = oracle.focus(_problem(sc, sc.api_arrays()), oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    assert np.all(np.isfinite(img))
    err = rel_l2(img[pix], ref)
    assert err <= tol, err


@pytest.mark.parametrize("shift,tol", FAR)
def test_map_coordinates_noalloc(cuda_device, shift, tol):
    import torch

    from test_zz_no_alloc import _noalloc_args, _noalloc_twice

    sc = _moved(shift, seed=9, n_pri=300, n_samples=256, nx=97, ny=83, spacing=1e-3)
    api = sc.api_arrays()
    a, keep = _noalloc_args(api, sc.grid, torch, pos64=sc.positions, grid64=sc.grid)
    got = _noalloc_twice(a)
    pix = np.unique(np.random.default_rng(5).choice(got.size, 60, replace=False))
    ref = oracle.focus(_problem(sc, api), oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    err = rel_l2(got[pix], ref)
    assert np.all(np.isfinite(got)) and err <= tol, err


def test_measured_geometry_does_not_depend_on_the_origin(cuda_device):
    """The direct kernels' plans: unit spans under a finite band (radii of the tiles) and anchored
    ranges (distance of pixels from their anchors) of a grid moved to map coordinates."""
    shift = FAR[0][0]
    kw = dict(seed=303, n_pri=600, n_samples=128, nx=64, ny=96, rail_len=0.6)
    spans = []
    for s in (0.0, shift):
        sc = _moved(s, **kw)
        api = sc.api_arrays()
        api["velocity"][..., 0] = 0.08
        p = _processor(sc, api, band=14.0)
        import torch

        p.focusDevice(torch.empty(p.numPixels(), dtype=torch.complex64, device="cuda"))
        p.check()
        st = p.lastStats()
        assert st["stage_samples"] > 0 and st["tile_cols"] == 16
        spans.append(st["span_permille"])
    assert spans[0] < 1000 and abs(spans[0] - spans[1]) <= 1
    sc = _moved(shift, seed=5, n_pri=256, n_samples=256, nx=64, ny=32, spacing=2e-3)
    p = _processor(sc)
    p.focusDevice(torch.empty(p.numPixels(), dtype=torch.complex64, device="cuda"))
    p.check()
    assert p.lastStats()["anchor_pixels"] == 32


def _banded(shift, **kw):
    sc = _moved(shift, **kw)
    api = sc.api_arrays()
    api["velocity"][..., 0] = 0.08
    return sc, api


@pytest.mark.parametrize("nx,ny,spacing,height,shift,anchored,group", [
    (57, 131, 1e-3, 0.1, KM, True, 8),
    (57, 131, 1e-3, 0.03, KM, False, 0),
    (64, 80, 8e-3, 0.05, KM, True, 2),
    (57, 131, 1e-3, 0.3, FAR[0][0], True, 8),
    (57, 131, 1e-3, 0.3, FAR[0][0], False, 0),
])
def test_far_grid_under_a_finite_band(cuda_device, nx, ny, spacing, height, shift, anchored, group):
    """Chirps are left out for a warp from its anchors' Doppler. Tolerance 2e-4, as for every finite band:
    a chirp at the inclusive edge may fall on either side in FP32 and FP64."""
    sc, api = _banded(shift, seed=nx + ny, n_pri=750, n_samples=192, nx=nx, ny=ny, spacing=spacing, height=height,
                      rail_len=0.75, y0=0.05)
    import _sarlabtdc

    p = _sarlabtdc.TdcProcessor(0)
    p.setSkipTest(False)  # (its points are FP32 by definition)
    p.setRawData(*api.values())
    p.setChirpPositionsF64(sc.positions)
    p.setFocusGridF64(sc.grid)
    p.setAnchoredRanges(anchored)
    p.prepare(0.0, 9.0, False, False, True)
    p.uploadGrid()
    img, anchor = _focus(p)
    assert anchor == group
    pix = np.unique(np.random.default_rng(5).choice(img.size, 150, replace=False))
    ref = oracle.focus(_problem(sc, api), oracle.Opts(applyRangeWin=False, dopplerBandwidth=9.0, skip_test=False),
                       pixels=pix)
    err = rel_l2(img[pix], ref)
    assert np.any(ref) and err <= 2e-4, err


@pytest.mark.parametrize("height,shift", [(0.03, KM), (0.3, FAR[0][0])])
def test_far_noalloc_under_a_finite_band(cuda_device, height, shift):
    import torch

    from test_zz_no_alloc import _noalloc_args, _noalloc_twice

    sc, api = _banded(shift, seed=12, n_pri=750, n_samples=192, nx=57, ny=131, spacing=1e-3, height=height, rail_len=0.75,
                      y0=0.05)
    a, keep = _noalloc_args(api, sc.grid, torch, pos64=sc.positions, grid64=sc.grid, band=9.0)
    got = _noalloc_twice(a)
    pix = np.unique(np.random.default_rng(5).choice(got.size, 150, replace=False))
    ref = oracle.focus(_problem(sc, api), oracle.Opts(applyRangeWin=False, dopplerBandwidth=9.0, skip_test=False),
                       pixels=pix)
    err = rel_l2(got[pix], ref)
    assert np.any(ref) and err <= 2e-4, err
