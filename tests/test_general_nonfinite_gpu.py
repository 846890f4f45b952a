"""The FP32 general kernel (csrc/tdc_general.cu) on a position that is not a number, under per-sample
windows that leave the chirp out of band."""
import numpy as np
import pytest

from test_general_window_gpu import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("sample", [1, 57, 99])
def test_non_finite_position_is_not_skipped(cuda_device, sample, uneven):
    """The phase of that sample is not a number at any pixel, in band or not."""
    import _sarlabtdc

    sc, api = _scene(64, 64, 100, 100, True, uneven, 0.02)
    pos = api["position"].copy()
    pos[0, sample, 1] = np.nan
    api["position"] = pos
    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    p.setFocusGrid(sc.grid.astype(np.float32))
    p.setSkipTest(False)
    p.start(0.0, 3.0, False, False, True)
    assert p.lastStats()["path_name"] == "general"
    assert np.all(np.isnan(p.getFocusedImage()))
