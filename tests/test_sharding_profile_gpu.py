"""Pixel sharding through range profiles, on grids whose row blocks have another geometry than the
whole grid: row spacing that grows, so that the first block alone could share anchors among more
pixels, and pixels jittered, so that no two blocks have the same reach. The blocks, planned for the
whole grid, assemble into its image bit for bit."""
import numpy as np
import pytest

from sarlabtdc import scenes, sharding

pytestmark = pytest.mark.gpu

INF = float("inf")


def _grid(kind, nx, ny, spacing):
    g = scenes.ground_grid(nx, ny, spacing, y0=0.1)
    if kind == "growing":
        g[..., 0] *= 1.0 + 1.5 * np.arange(ny)[:, None] / ny
    elif kind == "jittered":
        g += np.random.default_rng(5).uniform(-0.05 * spacing, 0.05 * spacing, g.shape)
    return g


@pytest.mark.parametrize("kind,nx,ny,n_pri,spacing,height,band,fp64,group", [
    ("growing", 64, 96, 700, 1e-3, 0.3, INF, True, 4),
    ("growing", 64, 96, 700, 1e-3, 0.3, 14.0, False, 4),
    ("growing", 300, 250, 820, 0.5e-3, 0.3, INF, False, 8),   # the first block alone: 16
    ("jittered", 64, 96, 700, 1e-3, 0.04, INF, True, 8),
    ("plane", 320, 256, 820, 1e-3, 0.2, INF, True, 16),
])
@pytest.mark.parametrize("world", [2, 3])
def test_blocks_of_any_geometry_assemble_the_whole_grid(cuda_device, kind, nx, ny, n_pri, spacing, height, band, fp64,
                                                        group, world):
    import _sarlabtdc

    sc = scenes.small_scene(seed=nx + n_pri, n_pri=n_pri, n_samples=128, nx=nx, ny=ny, rail_len=0.6, jitter=0.2e-3,
                            height=height, device="cuda")
    api = sc.api_arrays()
    api["velocity"][..., 0] = 0.08
    grid = _grid(kind, nx, ny, spacing)
    args = (0.0, band, False, True, True)

    def set_grid(p):
        if fp64:
            p.setChirpPositionsF64(sc.positions)
            p.setFocusGridF64(grid)
        else:
            p.setFocusGrid(grid.astype(np.float32))

    p = _sarlabtdc.TdcProcessor(0)
    p.setRawData(*api.values())
    set_grid(p)
    p.start(*args)
    st = p.lastStats()
    assert st["stage_samples"] == 0 and st["anchor_pixels"] == group
    whole = p.getFocusedImage()
    out = np.empty_like(whole)
    for rank in range(world):
        sp = sharding.ShardedProcessor(0, rank, world)
        sp.setRawData(*api.values())
        set_grid(sp)
        sp.start(*args)
        assert sp.proc.lastStats()["anchor_pixels"] == group
        r0, r1 = sp.rows
        out[r0:r1] = sp.getLocalImage()
    np.testing.assert_array_equal(out, whole)
