"""Histories that the fixed-point positions of the tabulated points do not hold, or whose points they cannot prove:
oblique lines over thin slices, lines that leave the grid through its zero corner, lines along voxel faces.
Their lists are the reference's, and they take no longer than without the table.
"""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P

pytestmark = pytest.mark.gpu


def config(thickness, **extra):
    return Config(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=thickness, RECON_CYL_RADIUS=10.0, COLUMNS=200, ROWS=200,
                  SLICES=int(8 / thickness), SSD_V_SIZE=9.0, DROP_BLOCK_SIZE=60000, HISTORIES_PER_BLOCK=0, LAMBDA=1e-4,
                  MLP_U_STEP=0.05, SCATTER_MODE="DETERMINISTIC", **extra)


def oblique(cfg, n, slope, seed=5):
    """Histories of the head phantom on lines through the middle plane, z = s u with |s| up to `slope`."""
    tr = P.simulate_tracks(P.head_phantom(), int(1.4 * n) + 1000, seed=seed, continuous_angles=True, t_extent=16.0, v_extent=6.8)
    h = {k: v.numpy()[:n].copy() for k, v in P.reconstruction_histories(cfg, tr).items()}
    assert len(h["WEPL"]) == n
    s = np.random.default_rng(seed).uniform(-slope, slope, n)
    u = np.hypot(h["x_exit"] - h["x_entry"], h["y_exit"] - h["y_entry"])
    h["z_entry"], h["z_exit"] = (-s * u / 2).astype(np.float32), (s * u / 2).astype(np.float32)
    h["xz_entry_angle"] = h["xz_exit_angle"] = np.arctan(s).astype(np.float32)
    v = [np.floor((a + 10) / 0.1) for a in (h["x_entry"], -h["y_entry"])] + [np.floor((4 - h["z_entry"]) / cfg.VOXEL_THICKNESS)]
    h["first_MLP_voxel"] = (v[0] + 200 * v[1] + 40000 * v[2]).astype(np.uint32)
    return h


def beyond(cfg, n, slope, seed=6):
    """Half of the oblique lines moved across the grid's zero corner, a quarter along the x axis on faces."""
    h = oblique(cfg, n, slope, seed)
    k = n // 2
    for f in ("x_entry", "x_exit"):
        h[f][:k] -= 7.0
    for f in ("y_entry", "y_exit"):
        h[f][:k // 2] += 7.0
    axis = slice(k, k + n // 4)
    for f in ("y_entry", "y_exit", "z_entry", "z_exit", "xy_entry_angle", "xy_exit_angle", "xz_entry_angle", "xz_exit_angle"):
        h[f][axis] = 0.0
    h["x_entry"][axis] = -8.0
    h["x_exit"][axis] = 8.0
    return h


@pytest.mark.parametrize("make", [oblique, beyond])
@pytest.mark.parametrize("thickness,slope", [(0.25, 0.18), (0.0625, 0.18), (0.03125, 0.18), (0.03125, 0.05)])
@pytest.mark.parametrize("threads", [64, 128, 256])
def test_lists_are_the_reference_order_ones(make, thickness, slope, threads):
    from pct_reconstruction_b200 import Context
    out = []
    for fast in (1, 0):
        cfg = config(thickness, EXACT_FAST_POINTS=fast, PATH_CTA_THREADS=threads)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(make(cfg, 20011, slope))
            ctx.x_host_2_GPU(np.full(cfg.NUM_VOXELS, 0.9, np.float32))
            ctx.DROP_full_tx_iteration(1)
            out.append((ctx.x_GPU_2_host(), ctx.counters()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]


def test_oblique_lines_over_thin_slices_take_no_longer():
    """The path kernel, against the one that computes every point in the reference's order."""
    from pct_reconstruction_b200 import Context
    ms = []
    for fast in (1, 0):
        cfg = config(0.0625, EXACT_FAST_POINTS=fast)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(oblique(cfg, 300_000, 0.18))
            ctx.x_host_2_GPU(np.full(cfg.NUM_VOXELS, 0.9, np.float32))
            for _ in range(3):
                ctx.DROP_full_tx_iteration(1)
            ms.append(np.median([ctx.profile_drop_iteration()["path"]["ms"] for _ in range(9)]))
    print(f"path kernel: tabulated {ms[0]:.3f} ms, reference order {ms[1]:.3f} ms")
    assert ms[0] < ms[1]
