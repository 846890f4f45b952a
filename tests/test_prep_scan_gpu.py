"""The scan that decides whether a per-sample trajectory varies within its chirps
(csrc/tdc_prep.cu): one differing float anywhere in the positions, velocities or attitudes is
found, and differences between chirps are not taken for one."""
import numpy as np
import pytest

from sarlabtdc import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pri,n_samples", [(3, 2), (5, 31), (7, 33), (64, 100), (130, 257), (33, 2000)])
def test_scan_finds_one_differing_float(cuda_device, n_pri, n_samples):
    import _sarlabtdc

    sc = scenes.small_scene(seed=1, n_pri=n_pri, n_samples=n_samples, nx=4, ny=4, spacing=1e-3, device="cuda")
    base = sc.api_arrays()
    vel = np.zeros_like(base["velocity"])
    vel[..., 0] = 0.05 + 1e-3 * np.arange(n_pri, dtype=np.float32)[:, None]
    base["velocity"] = vel
    p = _sarlabtdc.TdcProcessor(0)
    p.setFocusGrid(sc.grid.astype(np.float32))

    def variant(key=None, at=None):
        api = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in base.items()}
        if key:
            flat = api[key].reshape(-1)
            flat[at] = np.float32(flat[at] + np.float32(1e-3))
        p.setRawData(*api.values())
        p.start(0.0, 50.0, False, False, True)
        return p.lastStats()["general_variant"]

    assert variant() == 0
    rng = np.random.default_rng(2)
    for key, k, bit in (("position", 3, 1), ("velocity", 3, 2), ("attitude", 4, 2)):
        n = n_pri * n_samples * k
        spots = {0, k - 1, n - 1, n - k, (n_samples - 1) * k, n_samples * k, n_samples * k + k, 4 * (n // 4) - 1,
                 31 * 4, 31 * 4 - 1, 32 * 4 + 1, *rng.integers(0, n, 4).tolist()}
        for at in sorted(s for s in spots if 0 <= s < n):
            assert variant(key, at) & bit, (key, at)
