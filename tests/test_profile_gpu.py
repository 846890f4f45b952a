"""GPU parity of the focus through range profiles (csrc/tdc_profile.cu): focuses of at least
3e8 correlations read each (pixel, chirp) sum from a per-chirp table of the row's spectrum
instead of summing the samples. Checked on pixel subsets against the FP64 oracle, over the
forms the path takes: pixels sharing an anchor in groups of 8, 4, 2 and 1, ragged runs and
bands, one run, odd row lengths, double-float inputs, ranges too short for the range-difference
series, an antenna on a pixel, a falling chirp, rows beyond whole-row staging.

Tolerance: relative L2 <= 3e-6, from the parts of the error (each rms, radians of phase or
relative to the row): sample frequencies as an affine fit of FP32 sample times 1.5e-6,
interpolation 3e-7, phase difference from the anchor 1e-6 at 5 cycles, FP32 sums 5e-7,
sincos 3e-7."""
import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import rel_l2

pytestmark = pytest.mark.gpu

INF = float("inf")
L2_TOL = 3e-6


def _check(sc, group, pos64=None, grid64=False, anchored=True, api=None, seed=3):
    import _sarlabtdc

    api = sc.api_arrays() if api is None else api
    grid = sc.grid if grid64 else sc.grid.astype(np.float32)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    if pos64 is not None:
        p.setChirpPositionsF64(pos64)
    (p.setFocusGridF64 if grid64 else p.setFocusGrid)(grid)
    p.setAnchoredRanges(anchored)
    p.start(0.0, INF, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    # (rows are staged by the direct kernels only)
    assert st["path_name"] == "fp32_bulk" and st["stage_samples"] == 0
    assert st["anchor_pixels"] == (group if group > 1 else 0)
    n = img.size
    edge = [0, 7, 8, sc.grid.shape[1] - 1, sc.grid.shape[1] % n, n - 1]
    pix = np.unique(np.concatenate([edge, np.random.default_rng(seed).choice(n, 60, replace=False)]))
    prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"],
                          position=pos64 if pos64 is not None else api["position"], velocity=api["velocity"],
                          attitude=api["attitude"], modRate=api["modRate"], startFreq=api["startFreq"], grid=grid)
    ref = oracle.focus(prob, oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    assert np.all(np.isfinite(img))
    err = rel_l2(img[pix], ref)
    assert err <= L2_TOL, err
    return img


@pytest.mark.parametrize("nx,ny,n_pri,n_samples,spacing,group", [
    (57, 131, 300, 256, 1e-3, 8),     # ragged groups, a last band of 3 runs
    (8, 512, 1024, 128, 2e-3, 8),     # one group a run
    (129, 64, 129, 500, 2e-3, 8),     # one pixel more than whole groups, one chirp past a skip chunk
    (9000, 1, 150, 400, 0.2e-3, 8),   # one long run
    (70, 110, 256, 256, 3.9e-3, 4),
    (70, 110, 256, 256, 8e-3, 2),
    (70, 110, 256, 256, 2e-2, 1),
    (64, 65, 1000, 123, 1e-3, 8),     # odd row length, many chirps
    (256, 256, 40, 12345, 2e-3, 8),   # rows too long for whole-row stages
    (301, 200, 64, 160, 1e-3, 8),     # two blocks of chirp records
])
def test_profile_focus_against_the_oracle(cuda_device, nx, ny, n_pri, n_samples, spacing, group):
    sc = scenes.small_scene(seed=nx + n_samples, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing,
                            jitter=0.2e-3, device="cuda")
    _check(sc, group)


def test_profile_focus_double_float_inputs_and_no_anchors(cuda_device):
    """FP64 positions and grid; and every range in double-float with anchored ranges off."""
    sc = scenes.small_scene(seed=7, n_pri=320, n_samples=300, nx=83, ny=77, spacing=1.3e-3, jitter=0.5e-3,
                            device="cuda")
    a = _check(sc, 8, pos64=sc.positions, grid64=True)
    b = _check(sc, 0, pos64=sc.positions, grid64=True, anchored=False)
    assert rel_l2(a, b) <= 2 * L2_TOL


def test_profile_focus_at_short_ranges(cuda_device):
    """The antenna 2 cm above the grid's edge and, for one chirp, on a pixel (its window is zero
    there): every range is too short for the series of the range difference."""
    sc = scenes.small_scene(seed=8, n_pri=300, n_samples=256, nx=72, ny=110, height=0.02, y0=0.01, device="cuda")
    api = sc.api_arrays()
    api["position"] = np.array(api["position"])
    api["position"][150, :, :] = sc.grid.astype(np.float32)[40, 21]
    _check(sc, 8, api=api)


def test_profile_focus_of_a_falling_chirp(cuda_device):
    """81 to 77 GHz: the cells run backwards in range."""
    sc = scenes.small_scene(seed=9, n_pri=300, n_samples=256, nx=72, ny=110, device="cuda")
    rng = np.random.default_rng(10)
    sc.radar = scenes.Radar(f0=81e9, bandwidth=-4e9, n_samples=256)
    scenes.finish_raw(sc, scenes.simulate_raw(sc.positions, sc.targets, sc.amps, sc.radar, "cuda"), 20.0, rng)
    _check(sc, 8)


@pytest.mark.parametrize("nx,ny,spacing,group,taper,centre,band,skip", [
    (57, 131, 1e-3, 8, True, 0.0, 14.0, True),    # ragged groups, a partial last skip chunk
    (131, 57, 2e-3, 8, False, 3.0, 9.0, True),    # rectangular window off the centre
    (64, 80, 3.9e-3, 4, True, -2.0, 20.0, False),
    (64, 80, 8e-3, 2, False, 0.0, 30.0, True),
    (64, 80, 2e-2, 1, True, 0.0, 20.0, True),
    (72, 110, 1e-3, 8, True, 500.0, 5.0, True),   # every chirp out of band
])
def test_profile_focus_under_a_finite_band(cuda_device, nx, ny, spacing, group, taper, centre, band, skip):
    """Antenna moving along the rail; most chirps are out of band for a pixel. Tolerance 2e-4, as
    for the direct kernels: a chirp at the inclusive edge of the band may fall on either side in
    FP32 and FP64."""
    import _sarlabtdc

    sc = scenes.small_scene(seed=nx + ny, n_pri=750, n_samples=192, nx=nx, ny=ny, spacing=spacing, rail_len=0.75,
                            device="cuda")
    api = sc.api_arrays()
    vel = np.zeros_like(api["velocity"])
    vel[..., 0] = 0.08
    api["velocity"] = vel
    grid = sc.grid.astype(np.float32)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.setSkipTest(skip)
    p.start(centre, band, False, False, taper)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert st["path_name"] == "fp32_bulk" and st["stage_samples"] == 0
    assert st["anchor_pixels"] == (group if group > 1 else 0)
    pix = np.unique(np.concatenate([[0, nx - 1, nx, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 100, replace=False)]))
    prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=api["position"],
                          velocity=api["velocity"], attitude=api["attitude"], modRate=api["modRate"],
                          startFreq=api["startFreq"], grid=grid)
    ref = oracle.focus(prob, oracle.Opts(dopplerWinCenter=centre, dopplerBandwidth=band, applyRangeWin=False,
                                         dopplerWinTaper=taper, skip_test=skip), pixels=pix)
    if not np.any(ref):
        assert not np.any(img[pix])
    else:
        assert rel_l2(img[pix], ref) <= 2e-4


@pytest.mark.parametrize("nx,ny,spacing,group,band,anchored", [
    (57, 131, 1e-3, 8, INF, True),
    (64, 80, 3.9e-3, 4, INF, True),
    (64, 80, 8e-3, 2, INF, True),
    (64, 80, 1e-3, 1, INF, False),
    (57, 131, 1e-3, 8, 14.0, True),
    (64, 80, 1e-3, 1, 14.0, False),
])
def test_profile_adjoint_against_the_oracle(cuda_device, nx, ny, spacing, group, band, anchored):
    """Gradient of a real loss of the image for every chirp's position, at offsets from the base
    trajectory, with and without a forward before it: against the FP64 oracle to 3e-6 relative
    L2, as the image (its parts scale alike); under a finite band, where FP32 and FP64 can put a
    chirp on either side of the edge, against the direct adjoint of the grid's quarters (too small
    for profiles; the gradient is a sum over pixels) to twice that."""
    import torch

    import _sarlabtdc

    sc = scenes.small_scene(seed=nx + ny, n_pri=520, n_samples=192, nx=nx, ny=ny, spacing=spacing, rail_len=0.52,
                            jitter=0.2e-3, device="cuda")
    api = sc.api_arrays()
    vel = np.zeros_like(api["velocity"])
    vel[..., 0] = 0.08
    api["velocity"] = vel
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setChirpPositionsF64(sc.positions)
    p.setFocusGridF64(sc.grid)
    p.setAnchoredRanges(anchored)
    p.prepare(0.0, band, False, False, True)
    p.uploadGrid()
    p.keepChirpSums(True)
    rng = np.random.default_rng(11)
    off = rng.normal(0, 0.1e-3, (sc.n_pri, 3))
    g = (rng.normal(size=nx * ny) + 1j * rng.normal(size=nx * ny)).astype(np.complex64)
    off_d, g_d = torch.from_numpy(off).cuda(), torch.from_numpy(g).cuda()
    p.setChirpOffsetsDevice(off_d)
    grad = torch.empty((sc.n_pri, 3), dtype=torch.float64, device="cuda")
    p.adjointDevice(g_d, grad)
    alone = grad.cpu().numpy()
    img = torch.empty(nx * ny, dtype=torch.complex64, device="cuda")
    p.focusDevice(img)
    assert p.lastStats()["anchor_pixels"] == (group if group > 1 else 0)
    p.adjointDevice(g_d, grad)
    assert p.lastStats()["adjoint_stored"] == 0
    np.testing.assert_array_equal(grad.cpu().numpy(), alone)
    if np.isinf(band):
        prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=sc.positions,
                              velocity=vel[:, 0, :], modRate=api["modRate"], startFreq=api["startFreq"], grid=sc.grid)
        ref = oracle.adjoint_offsets(prob, oracle.Opts(applyRangeWin=False), off, g.astype(np.complex128))
        assert rel_l2(alone, ref) <= 3e-6
        return
    ref = np.zeros_like(alone)
    for k in range(4):
        rows = slice(k * ny // 4, (k + 1) * ny // 4)
        part = np.ascontiguousarray(sc.grid[rows])
        p.setFocusGridF64(part)
        p.uploadGrid()
        g_part = torch.from_numpy(np.ascontiguousarray(g.reshape(ny, nx)[rows].ravel())).cuda()
        p.adjointDevice(g_part, grad)
        ref += grad.cpu().numpy()
    assert rel_l2(alone, ref) <= 6e-6


@pytest.mark.parametrize("nx,ny,n_pri,n_samples,spacing,drift,accel", [
    (57, 131, 300, 256, 1e-3, 0.3e-3, 0.0),
    (131, 57, 129, 777, 1e-3, 0.5e-3, 0.0),
    (64, 80, 400, 300, 2e-3, 0.2e-3, 0.0),
    (64, 80, 400, 300, 3.9e-3, 0.3e-3, 0.0),
    (64, 80, 400, 300, 2e-2, 0.3e-3, 0.0),
    (57, 131, 300, 256, 1e-3, 0.2e-3, 1e-6),   # a little acceleration
])
def test_profile_focus_of_smooth_motion(cuda_device, nx, ny, n_pri, n_samples, spacing, drift, accel):
    """Positions moving within each chirp, at least 3e8 correlations. The oracle reads every
    sample's FP32 position; the fit smooths their rounding, 1.7e-8 m rms a coordinate or 5e-5 rad
    a sample, which the sum over samples averages: tolerance 2e-5. The FP32 general kernel, which
    follows each position, and this path agree to the same."""
    import _sarlabtdc

    sc = scenes.small_scene(seed=nx + n_samples, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing,
                            rail_len=0.3, device="cuda")
    rng = np.random.default_rng(4)
    api = sc.api_arrays()
    u = (np.arange(n_samples) / n_samples)[None, :, None]
    pos = api["position"].astype(np.float64) + u * rng.normal(0.0, drift, (n_pri, 1, 3))
    pos = pos + u * u * rng.normal(0.0, accel, (n_pri, 1, 3)) if accel else pos
    api["position"] = pos.astype(np.float32)
    grid = sc.grid.astype(np.float32)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.start(0.0, INF, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert st["path_name"] == "fp32_motion" and st["stage_samples"] == 0 and st["motion_segment"] == 0
    pix = np.unique(np.concatenate([[0, nx - 1, nx, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 60, replace=False)]))
    prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=api["position"],
                          velocity=api["velocity"], attitude=api["attitude"], modRate=api["modRate"],
                          startFreq=api["startFreq"], grid=grid)
    ref = oracle.focus(prob, oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    err = rel_l2(img[pix], ref)
    assert err <= 2e-5, err
    p.setMotionPath(False)
    p.start(0.0, INF, False, False, True)
    assert p.lastStats()["path_name"] == "general"
    assert rel_l2(img, p.getFocusedImage().ravel()) <= 2e-5


@pytest.mark.parametrize("nx,ny,n_pri,n_samples,spacing,amp,anchored", [
    (57, 131, 300, 256, 1e-3, 20e-6, True),
    (131, 57, 129, 777, 2e-3, 10e-6, True),
    (70, 110, 256, 256, 3.9e-3, 20e-6, True),
    (70, 110, 256, 256, 8e-3, 20e-6, True),
    (57, 131, 300, 256, 1e-3, 20e-6, False),
    (57, 131, 300, 256, 1e-3, 90e-6, True),   # beyond the series: the direct kernel
])
def test_profile_focus_of_vibration(cuda_device, nx, ny, n_pri, n_samples, spacing, amp, anchored):
    """An antenna that vibrates within each chirp, in a direction of each chirp's own, beside a
    constant velocity. Every sample's FP32 position counts, as in the direct kernel. Tolerance 5e-6:
    the 3e-6 above, 5e-7 of the series in the deviations, and at most 4.5e-6 at the edge of a group
    (1.5e-6 rms) of the directions' second order."""
    import _sarlabtdc

    sc = scenes.small_scene(seed=nx + n_samples, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing,
                            rail_len=0.3, device="cuda")
    rng = np.random.default_rng(6)
    api = sc.api_arrays()
    u = (np.arange(n_samples) / n_samples)[None, :, None]
    along = rng.normal(size=(n_pri, 1, 3))
    along /= np.linalg.norm(along, axis=2, keepdims=True)
    pos = api["position"].astype(np.float64) + u * rng.normal(0.0, 0.2e-3, (n_pri, 1, 3))
    pos = pos + amp * along * (0.7 * np.sin(2 * np.pi * 3 * u + rng.uniform(0, 2 * np.pi, (n_pri, 1, 1)))
                               + 0.3 * np.sin(2 * np.pi * 11 * u))
    api["position"] = pos.astype(np.float32)
    grid = sc.grid.astype(np.float32)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.setAnchoredRanges(anchored)
    p.start(0.0, INF, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert st["path_name"] == "general" and (st["stage_samples"] == 0) == (amp < 50e-6)
    if not anchored:
        assert st["anchor_pixels"] == 0
    pix = np.unique(np.concatenate([[0, nx - 1, nx, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 60, replace=False)]))
    prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=api["position"],
                          velocity=api["velocity"], attitude=api["attitude"], modRate=api["modRate"],
                          startFreq=api["startFreq"], grid=grid)
    ref = oracle.focus(prob, oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    err = rel_l2(img[pix], ref)
    assert err <= 5e-6, err


def _axis_grid(sc, axis):
    """The scene's ground plane with its runs along x, or its rows and columns exchanged (along y)."""
    return sc.grid if axis == 0 else np.ascontiguousarray(sc.grid.transpose(1, 0, 2))


@pytest.mark.parametrize("nx,ny,n_pri,spacing,height,axis,group", [
    (333, 200, 1000, 1e-3, 0.3, 0, 16),   # ragged groups, a last band of runs, 1.3 groups a tile
    (200, 333, 1000, 1e-3, 0.3, 1, 16),   # runs along y
    (320, 256, 800, 0.7e-3, 0.12, 0, 16),  # ranges from 0.12 m: the long series
    (256, 320, 800, 1e-3, 0.03, 1, 16),   # ranges too short for any series
    (256, 320, 800, 1.5e-3, 0.3, 0, 8),   # 16 span too many cycles
    (75, 130, 200, 1e-3, 0.3, 1, 8),      # too few pairs
    (75, 130, 200, 1e-3, 0.02, 1, 8),
])
def test_profile_focus_of_runs_along_an_axis(cuda_device, nx, ny, n_pri, spacing, height, axis, group):
    """Tolerance 4e-6: the 3e-6 above, and 1.5e-6 of phases at up to 4.5 cycles unreduced."""
    import _sarlabtdc

    sc = scenes.small_scene(seed=nx + n_pri, n_pri=n_pri, n_samples=160, nx=nx, ny=ny, spacing=spacing, height=height,
                            y0=0.02 if height < 0.2 else 0.2, device="cuda")
    api = sc.api_arrays()
    grid = _axis_grid(sc, axis).astype(np.float32)
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(grid)
    p.start(0.0, INF, False, False, True)
    img, st = p.getFocusedImage().ravel(), p.lastStats()
    assert st["stage_samples"] == 0 and st["anchor_pixels"] == group
    cols = grid.shape[1]
    pix = np.unique(np.concatenate([[0, 15, 16, cols - 1, cols, img.size - 1],
                                    np.random.default_rng(5).choice(img.size, 60, replace=False)]))
    prob = oracle.Problem(raw=api["rawData"], sampleTimes=api["sampleTimes"], position=api["position"],
                          velocity=api["velocity"], attitude=api["attitude"], modRate=api["modRate"],
                          startFreq=api["startFreq"], grid=grid)
    ref = oracle.focus(prob, oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF), pixels=pix)
    assert np.all(np.isfinite(img))
    err = rel_l2(img[pix], ref)
    assert err <= 4e-6, err


@pytest.mark.parametrize("axis,band,n_pri", [(0, INF, 1000), (1, INF, 1000), (1, INF, 300), (0, 14.0, 300), (1, 14.0, 300)])
def test_profile_adjoint_of_runs_along_an_axis(cuda_device, axis, band, n_pri):
    """Groups of 16 and 8 against every pixel's range in double-float (checked against the oracle
    above): 4e-6 and 3e-6 of either, relative L2 7e-6."""
    import torch

    import _sarlabtdc

    sc = scenes.small_scene(seed=31, n_pri=n_pri, n_samples=160, nx=301, ny=210, spacing=1e-3, rail_len=0.5,
                            jitter=0.2e-3, device="cuda")
    api = sc.api_arrays()
    vel = np.zeros_like(api["velocity"])
    vel[..., 0] = 0.08
    api["velocity"] = vel
    grid = _axis_grid(sc, axis)
    n = grid.shape[0] * grid.shape[1]
    rng = np.random.default_rng(12)
    g_d = torch.from_numpy((rng.normal(size=n) + 1j * rng.normal(size=n)).astype(np.complex64)).cuda()
    grads = []
    for anchored in (True, False):
        p = _sarlabtdc.TdcProcessor(0)
        p.setRawData(*api.values())
        p.setChirpPositionsF64(sc.positions)
        p.setFocusGridF64(grid)
        p.setAnchoredRanges(anchored)
        p.prepare(0.0, band, False, False, True)
        p.uploadGrid()
        grad = torch.empty((sc.n_pri, 3), dtype=torch.float64, device="cuda")
        p.adjointDevice(g_d, grad)
        grads.append(grad.cpu().numpy())
    assert np.all(np.isfinite(grads[0])) and np.any(grads[0])
    assert rel_l2(grads[0], grads[1]) <= (7e-6 if np.isinf(band) else 4e-4)
