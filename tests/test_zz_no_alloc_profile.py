"""GPU parity of tdc_focus_noalloc where it may take range profiles (at least 3e8 correlations):
the form is decided on the device from the grid and the trajectory. Tables that fit the fixed
scratch, a finite band with skip points, double-float inputs, and a captured call replayed on a
grid changed in place so that its table does not fit and the direct form is taken. Tolerances: relative L2 <= 3e-6 against the FP64 oracle as for the processor's
range profiles, 2e-4 under a finite band (chirps at its edge)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import problem_from_api, rel_l2
from test_zz_no_alloc import _noalloc_args, _noalloc_twice

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("nx,ny,n_pri,n_samples,spacing,band,fp64", [
    (100, 80, 300, 256, 2e-3, INF, False),
    (97, 83, 300, 256, 1e-3, INF, True),
    (8, 700, 750, 150, 1e-3, 18.0, False),
])
def test_noalloc_large_calls_against_the_oracle(cuda_device, nx, ny, n_pri, n_samples, spacing, band, fp64):
    import torch

    sc = scenes.small_scene(seed=nx + n_samples, n_pri=n_pri, n_samples=n_samples, nx=nx, ny=ny, spacing=spacing,
                            rail_len=0.6, jitter=0.2e-3 if fp64 else 0.0, device="cuda")
    api = sc.api_arrays()
    finite = np.isfinite(band)
    if finite:
        vel = np.zeros_like(api["velocity"])
        vel[..., 0] = 0.2
        api["velocity"] = vel
    a, keep = _noalloc_args(api, sc.grid, torch, pos64=sc.positions if fp64 else None,
                            grid64=sc.grid if fp64 else None, centre=2.0 if finite else 0.0, band=band, skip=finite)
    got = _noalloc_twice(a)
    pix = np.unique(np.concatenate([[0, nx - 1, nx, got.size - 1],
                                    np.random.default_rng(5).choice(got.size, 60, replace=False)]))
    prob = problem_from_api(api, sc.grid, pos64=sc.positions if fp64 else None, grid64=fp64)
    ref = oracle.focus(prob, oracle.Opts(dopplerWinCenter=2.0 if finite else 0.0, dopplerBandwidth=band,
                                         applyRangeWin=False, dopplerWinTaper=True, skip_test=finite), pixels=pix)
    assert np.all(np.isfinite(got)) and np.abs(ref).max() > 0
    assert rel_l2(got[pix], ref) <= (2e-4 if finite else 3e-6)


def test_noalloc_captured_call_takes_either_form(cuda_device):
    """One captured call: replayed on its grid (profiles) it gives the blocking call's image bit
    for bit; with a few grid points moved 20 m away in place the table no longer fits and the
    direct form runs, the other pixels agreeing to FP32 rounding; moved back, the first image."""
    import torch

    import _tdc_capi

    lib = _tdc_capi.lib()
    sc = scenes.small_scene(seed=62, n_pri=300, n_samples=256, nx=100, ny=80, device="cuda")
    a, keep = _noalloc_args(sc.api_arrays(), sc.grid, torch)
    grid = keep[2]
    first = _noalloc_twice(a)
    out = torch.empty(a.n_pix, dtype=torch.complex64, device="cuda")
    status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc = lib.tdc_focus_noalloc_async(C.byref(a), C.c_void_p(out.data_ptr()), C.c_void_p(status.data_ptr()),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, _tdc_capi.last_error()

    def replay():
        status.fill_(-1)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        return out.cpu().numpy()

    np.testing.assert_array_equal(replay(), first)
    kept = grid[:4].clone()
    grid[:4, 1] += 20.0
    moved = replay()
    assert rel_l2(moved[4:], first[4:]) <= 6e-6 and not np.array_equal(moved[4:], first[4:])
    grid[:4] = kept
    np.testing.assert_array_equal(replay(), first)
