"""The path kernel's tabulated MLP points (EXACT_FAST_POINTS = 1) against reference-order points.

With the deterministic scatter two iterations give bit-identical images if, and only if (up to a
coincidence), every voxel list, chord and path length agrees, so the images and the diagnostic
counters of EXACT_FAST_POINTS = 1 and 0 must be equal.  The cases are the edges of the table's range:
MLP steps that are and are not whole lookup-table steps, several buckets per step, grids whose
positions need fewer fraction bits, one history, warps with one history, histories so short that they
have no row, along the axes, outside the grid, and with angles far larger than a scan's.
"""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P

GRID = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=6.4, SSD_V_SIZE=5.0,
            DROP_BLOCK_SIZE=10000, HISTORIES_PER_BLOCK=0, SCATTER_MODE="DETERMINISTIC", MIN_MLP_LENGTH=2)


def simulated(cfg, n, seed):
    tr = P.simulate_tracks(P.water_cylinder_phantom(0.94 * cfg.RECON_CYL_RADIUS), int(1.6 * n) + 200, seed=seed,
                           continuous_angles=True, t_extent=1.8 * cfg.RECON_CYL_RADIUS,
                           v_extent=0.85 * cfg.RECON_CYL_HEIGHT, span=cfg.RECON_CYL_RADIUS)
    return {k: v.numpy()[:n] for k, v in P.reconstruction_histories(cfg, tr).items()}


def irregular(cfg, n, seed):
    """Histories no scan produces but the entry points accept: any two points in and around the grid,
    any angles, zero length, exactly along an axis, on voxel faces."""
    rng = np.random.default_rng(seed)
    R, H = cfg.RECON_CYL_RADIUS, cfg.RECON_CYL_HEIGHT
    h = {k: rng.uniform(-1.2 * R, 1.2 * R, n).astype(np.float32) for k in ("x_entry", "y_entry", "x_exit", "y_exit")}
    h.update({k: rng.uniform(-0.6 * H, 0.6 * H, n).astype(np.float32) for k in ("z_entry", "z_exit")})
    a = np.arctan2(h["y_exit"] - h["y_entry"], h["x_exit"] - h["x_entry"])
    h["xy_entry_angle"] = (a + rng.normal(0, 0.2, n)).astype(np.float32)
    h["xy_exit_angle"] = (a + rng.normal(0, 0.2, n)).astype(np.float32)
    h["xz_entry_angle"], h["xz_exit_angle"] = (rng.normal(0, 0.2, n).astype(np.float32) for _ in range(2))
    k = n // 8
    h["x_exit"][:k], h["y_exit"][:k] = h["x_entry"][:k], h["y_entry"][:k]  # zero length
    short = slice(k, 2 * k)  # a few steps long
    h["x_exit"][short] = h["x_entry"][short] + rng.uniform(-0.4, 0.4, k).astype(np.float32)
    h["y_exit"][short] = h["y_entry"][short]
    axis = slice(2 * k, 3 * k)  # along x on voxel faces, all angles 0
    for f in ("y_entry", "y_exit", "z_entry", "z_exit"):
        h[f][axis] = 0.0
    for f in ("xy_entry_angle", "xy_exit_angle", "xz_entry_angle", "xz_exit_angle"):
        h[f][axis] = 0.0
    h["WEPL"] = rng.uniform(0, 20, n).astype(np.float32)
    h["first_MLP_voxel"] = rng.integers(0, cfg.NUM_VOXELS, n).astype(np.uint32)
    return h


def both(params, make, n, seed):
    from pct_reconstruction_b200 import Context
    out = []
    for fast in (1, 0):
        cfg = Config(**params, EXACT_FAST_POINTS=fast)
        h = make(cfg, n, seed)
        x0 = np.linspace(0.5, 1.5, cfg.NUM_VOXELS, dtype=np.float32)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(h)
            ctx.x_host_2_GPU(x0)
            ctx.DROP_full_tx_iteration(1)
            x = ctx.x_GPU_2_host()
            counters = ctx.counters()
            counters.pop("wait_expired")
        assert np.any(x != x0) or n < 40
        out.append((x, counters))
    (x1, c1), (x0, c0) = out
    np.testing.assert_array_equal(x1, x0)
    assert c1 == c0


@pytest.mark.gpu
@pytest.mark.parametrize("step", [0.03125, 0.05, 0.051, 0.0333217, 0.1, 0.1270001, 0.4])
def test_steps(step):
    both(dict(GRID, MLP_U_STEP=step), simulated, 60000, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 129, 10001])
def test_counts(n):
    both(GRID, simulated, n, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [dict(VOXEL_WIDTH=0.02, VOXEL_HEIGHT=0.02, MLP_U_STEP=0.05),  # 640 voxels across
                                  dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.025, VOXEL_THICKNESS=0.05),
                                  dict(RECON_CYL_RADIUS=1.0, SSD_V_SIZE=1.5)])
def test_grids(grid):
    both(dict(GRID, **grid), simulated, 40000, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("per_block,order", [(640, 0), (0, 4096), (7, 16384)])
def test_blocks_and_order(per_block, order):
    both(dict(GRID, DROP_BLOCK_SIZE=3201, HISTORIES_PER_BLOCK=per_block, PATH_ORDER_WINDOW=order), simulated, 20011, 4)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [64, 128, 256])
def test_irregular_histories(threads):
    both(dict(GRID, PATH_CTA_THREADS=threads), irregular, 40000, 5)


@pytest.mark.gpu
def test_mixed_mode_takes_the_exact_lists():
    """With the table, PRECISION = MIXED walks the same points, so its lists are the exact mode's."""
    from pct_reconstruction_b200 import Context
    out = []
    for precision in ("EXACT", "MIXED"):
        cfg = Config(**GRID, PRECISION=precision)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(simulated(cfg, 20000, 6))
            ctx.x_host_2_GPU(np.ones(cfg.NUM_VOXELS, np.float32))
            out.append(ctx.mlp_paths())
            ctx.DROP_full_tx_iteration(1)
            out[-1] += (ctx.x_GPU_2_host(),)
    for a, b in zip(out[0][:4], out[1][:4]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_allclose(out[1][4], out[0][4], rtol=0, atol=1e-6)  # FP32 updates of about 1e-4
