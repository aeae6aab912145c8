"""Path kernels of contexts without the table of MLP weights: EXACT_FAST_POINTS = 0, and grids too large for its
fixed-point positions (from about 1024 x 1024 columns and rows on).

The lists compared are those that the path kernels stored, as the export writes them.
"""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P

pytestmark = pytest.mark.gpu

SMALL = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=6.4, SSD_V_SIZE=5.0,
             DROP_BLOCK_SIZE=10000, HISTORIES_PER_BLOCK=0, MLP_U_STEP=0.05)
LARGE = dict(VOXEL_WIDTH=12.8 / 1100, VOXEL_HEIGHT=12.8 / 1100, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=6.4, COLUMNS=1100,
             ROWS=1100, SLICES=2, SSD_V_SIZE=1.5, DROP_BLOCK_SIZE=10000, HISTORIES_PER_BLOCK=0, MLP_U_STEP=0.05)


def histories(cfg, n, seed):
    tr = P.simulate_tracks(P.water_cylinder_phantom(6.0), 2 * n, seed=seed, continuous_angles=True, t_extent=11.5,
                           v_extent=0.85 * cfg.RECON_CYL_HEIGHT, span=6.4)
    h = {k: v.numpy()[:n] for k, v in P.reconstruction_histories(cfg, tr).items()}
    assert len(h["WEPL"]) == n
    return h


def stored_lists(params, n, where, iterations=0):
    """(voxel list per history, chords, image after `iterations`, counters) of one context."""
    from pct_reconstruction_b200 import Context
    cfg = Config(**params)
    where.mkdir()
    with Context(cfg) as ctx:
        ctx.set_reconstruction_histories(histories(cfg, n, 5))
        ctx.x_host_2_GPU(np.full(cfg.NUM_VOXELS, 0.9, np.float32))
        ctx.export_preprocessed(where)
        for k in range(iterations):
            ctx.DROP_full_tx_iteration(k + 1)
        image, counters = ctx.x_GPU_2_host(), ctx.counters()
    counts = np.fromfile(where / "voxels_per_path.bin", np.uint32)[1:]
    voxels = np.fromfile(where / "MLP_paths.bin", np.uint32)[1:]
    chords = np.frombuffer((where / "avg_chord_lengths.bin").read_bytes()[4:], np.float64)
    return np.split(voxels, np.cumsum(counts)[:-1]), chords, image, counters


def differing(a, b):
    return np.mean([not np.array_equal(x, y) for x, y in zip(a, b)])


@pytest.mark.parametrize("grid", [SMALL, LARGE])
@pytest.mark.parametrize("threads", [64, 128, 256])
def test_exact_lists_with_and_without_certain_points(grid, threads, tmp_path):
    """Tabulated points (small grid) and guarded points (large grid) against the reference's order."""
    grid = dict(grid, PATH_CTA_THREADS=threads, SCATTER_MODE="DETERMINISTIC")
    a = stored_lists(dict(grid, EXACT_FAST_POINTS=1), 20011, tmp_path / "a", iterations=2)
    b = stored_lists(dict(grid, EXACT_FAST_POINTS=0), 20011, tmp_path / "b", iterations=2)
    assert differing(a[0], b[0]) == 0
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[2], b[2])
    assert a[3] == b[3] and a[3]["path_overflow"] == 0


@pytest.mark.parametrize("precision", ["MIXED", "MIXED_COMPENSATED"])
@pytest.mark.parametrize("grid,fast", [(SMALL, 0), (LARGE, 0), (LARGE, 1)])
def test_mixed_lists_of_fp32_points(grid, fast, precision, tmp_path):
    """FP32 points: almost all lists are the exact ones, not all are (so the FP32 kernel ran), chords and
    lists agree with those of pct_mlp_paths, and images stay within the mixed modes' bar."""
    from pct_reconstruction_b200 import Context
    a = stored_lists(dict(grid, EXACT_FAST_POINTS=0), 20011, tmp_path / "a", iterations=2)
    b = stored_lists(dict(grid, EXACT_FAST_POINTS=fast, PRECISION=precision), 20011, tmp_path / "b", iterations=2)
    assert 0 < differing(a[0], b[0]) < 0.01 * (1 if grid is SMALL else 8.6)  # as many more steps near a face
    np.testing.assert_array_equal(a[1], b[1])
    rel = np.sqrt(np.mean((a[2].astype(np.float64) - b[2]) ** 2)) / np.sqrt(np.mean(a[2].astype(np.float64) ** 2))
    assert rel < 1e-4
    cfg = Config(**grid, EXACT_FAST_POINTS=fast, PRECISION=precision)
    with Context(cfg) as ctx:
        ctx.set_reconstruction_histories(histories(cfg, 20011, 5))
        counts, voxels, _, _ = ctx.mlp_paths(0, 3000)
    for k in range(3000):
        np.testing.assert_array_equal(voxels[k, :counts[k]], b[0][k])
