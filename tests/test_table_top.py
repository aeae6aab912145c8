"""Histories near the top of the grid, whose paths leave it there for some steps: the reference mirrors the slice
index (|z - zero|), and the tabulated points do so too.  Any scan that is wider than the reconstructed height
has them."""
import time

import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P

pytestmark = pytest.mark.gpu

GRID = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=6.4, SSD_V_SIZE=5.0,
            DROP_BLOCK_SIZE=3200, HISTORIES_PER_BLOCK=640, MLP_U_STEP=0.1)


def histories(cfg, n, top):
    """Of a scan as high as the grid; with `top`, those that enter or leave within 1 mm of its top only."""
    have, parts, seed = 0, [], 0
    while have < n:
        tr = P.simulate_tracks(P.water_cylinder_phantom(6.0), 400_000, seed=seed, device="cuda", t_extent=18.0, v_extent=4.0)
        h = P.reconstruction_histories(cfg, tr)
        if top:
            keep = (2.0 - h["z_entry"]).minimum(2.0 - h["z_exit"]) < 0.1
            h = {k: v[keep] for k, v in h.items()}
        parts.append({k: v.cpu().numpy() for k, v in h.items()})
        have += len(parts[-1]["WEPL"])
        seed += 1
    return {k: np.concatenate([p[k] for p in parts])[:n] for k in parts[0]}


@pytest.mark.parametrize("step", [0.05, 0.1])
@pytest.mark.parametrize("thickness", [0.25, 0.0625])
def test_lists_at_the_top(step, thickness):
    from pct_reconstruction_b200 import Context
    out = []
    for fast in (1, 0):
        cfg = Config(**dict(GRID, MLP_U_STEP=step, VOXEL_THICKNESS=thickness, SLICES=int(4 / thickness), DROP_BLOCK_SIZE=5000,
                            HISTORIES_PER_BLOCK=0, SCATTER_MODE="DETERMINISTIC"), EXACT_FAST_POINTS=fast)
        h = histories(cfg, 20011, top=True)
        v = np.floor((2 - h["z_entry"]) / cfg.VOXEL_THICKNESS)
        h["first_MLP_voxel"] = (h["first_MLP_voxel"].astype(np.int64) % (cfg.COLUMNS * cfg.ROWS) + cfg.COLUMNS * cfg.ROWS * v).astype(np.uint32)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(h)
            ctx.x_host_2_GPU(np.full(cfg.NUM_VOXELS, 0.9, np.float32))
            ctx.DROP_full_tx_iteration(1)
            out.append((ctx.x_GPU_2_host(), ctx.counters()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]


def test_scan_as_high_as_the_grid_takes_no_longer():
    """An iteration in chunks of 16 blocks, against one that computes every point in the reference's order."""
    from pct_reconstruction_b200 import Context
    ms = []
    for fast in (1, 0):
        cfg = Config(**GRID, EXACT_FAST_POINTS=fast)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(histories(cfg, 300_000, top=False))
            ctx.x_host_2_GPU(np.full(cfg.NUM_VOXELS, 0.9, np.float32))
            times = []
            for _ in range(15):
                t = time.perf_counter()
                ctx.DROP_full_tx_iteration(1)
                ctx.synchronize()
                times.append(time.perf_counter() - t)
            ms.append(1e3 * np.median(times[4:]))
    print(f"iteration: tabulated {ms[0]:.3f} ms, reference order {ms[1]:.3f} ms")
    assert ms[0] < ms[1]
