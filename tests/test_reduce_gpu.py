"""GPU parity of the partial-sum reductions (csrc/tdc_focus.cu): one thread a pixel for a few
chirp groups, sliced over a block's threads for many, at pixel counts either side of a
block. The groups are the planner's, about one per chirp for grids of a few tiles. Tolerance:
relative L2 <= 3e-6 (the FP32-bulk kernel's own error is 1e-6; the sums are FP64)."""
import numpy as np
import pytest

import oracle
from sarlabtdc import scenes
from tdc_testutil import problem_from_api, rel_l2, run_engine

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("nx,ny,n_pri", [(1, 1, 300), (31, 1, 15), (32, 1, 16), (33, 1, 17), (11, 3, 129), (8, 8, 1000),
                                         (70, 60, 2)])
def test_reduction_over_chirp_groups(cuda_device, nx, ny, n_pri):
    sc = scenes.small_scene(seed=nx + n_pri, n_pri=n_pri, n_samples=64, nx=nx, ny=ny, jitter=0.2e-3, device="cuda")
    api = sc.api_arrays()
    img, _, _ = run_engine(api, sc.grid, (0.0, INF, False, False, True))
    ref = oracle.focus(problem_from_api(api, sc.grid), oracle.Opts(applyRangeWin=False, dopplerBandwidth=INF))
    assert np.abs(ref).max() > 0
    assert rel_l2(img, ref) <= 3e-6
