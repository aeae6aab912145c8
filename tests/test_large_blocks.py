"""DROP blocks on both sides of the lines from which a block takes more warps per SM instead of list entries in
registers (64 histories per SM for FP32 updates, 256 for double), with lists shorter and longer than the
registers hold then (4 entries per lane: 128 voxels).

Against the order-independent scatter.  One iteration from a smooth image: a voxel's update is the mean of at
most 2^11 float terms below 1e-2, summed in float (2^11 * 2^-24 * 1e-2 = 1.2e-6 per block, averaged over
the terms again), and x is rounded once per block: atol 2e-6 for two blocks.
"""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["EXACT", "MIXED"])
@pytest.mark.parametrize("per_sm,offset", [(64, -1), (64, 0), (256, -1), (256, 0)])
@pytest.mark.parametrize("columns,voxel", [(60, 0.2), (240, 0.08)])
def test_block_sizes(precision, per_sm, offset, columns, voxel):
    import torch
    from pct_reconstruction_b200 import Context
    block = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + offset
    p = dict(COLUMNS=columns, ROWS=columns, SLICES=8, VOXEL_WIDTH=voxel, VOXEL_HEIGHT=voxel, VOXEL_THICKNESS=0.4,
             RECON_CYL_RADIUS=columns * voxel / 2, SSD_V_SIZE=4.2, DROP_BLOCK_SIZE=block, HISTORIES_PER_BLOCK=0,
             LAMBDA=0.01, MLP_U_STEP=voxel / 2, PRECISION=precision)
    out = []
    for scatter in ("ATOMIC", "DETERMINISTIC"):
        cfg = Config(**p, SCATTER_MODE=scatter)
        R = cfg.RECON_CYL_RADIUS
        tr = P.simulate_tracks(P.water_cylinder_phantom(0.8 * R), 3 * block, seed=2, device="cuda", t_extent=1.8 * R,
                               v_extent=2.4)
        hist = {k: v[:block + 333].contiguous() for k, v in P.reconstruction_histories(cfg, tr).items()}
        assert len(hist["WEPL"]) == block + 333
        x0 = (0.95 + 0.1 * np.random.default_rng(3).random(cfg.NUM_VOXELS)).astype(np.float32)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(hist)
            ctx.x_host_2_GPU(x0)
            ctx.DROP_full_tx_iteration(1)
            out.append(ctx.x_GPU_2_host())
            lists = ctx.mlp_paths(0, 1000)[0]
            assert lists.max() > 128 if columns == 240 else lists.max() < 128
    assert np.count_nonzero(np.abs(out[0] - x0) > 1e-5) > 1000
    np.testing.assert_allclose(out[0], out[1], rtol=0, atol=2e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("slices", [1, 7])
def test_odd_number_of_voxels(slices):
    """The image updates take two voxels at a time; both scatters agree to the same tolerance."""
    from pct_reconstruction_b200 import Context
    p = dict(COLUMNS=65, ROWS=65, SLICES=slices, VOXEL_WIDTH=0.2, VOXEL_HEIGHT=0.2, VOXEL_THICKNESS=0.4, RECON_CYL_RADIUS=6.5,
             SSD_V_SIZE=0.4 * slices + 1.0, DROP_BLOCK_SIZE=300, HISTORIES_PER_BLOCK=0, LAMBDA=0.01, MLP_U_STEP=0.1)
    out = []
    for scatter in ("ATOMIC", "DETERMINISTIC"):
        cfg = Config(**p, SCATTER_MODE=scatter)
        tr = P.simulate_tracks(P.water_cylinder_phantom(5.0), 20000, seed=9, t_extent=10.0, v_extent=0.3 * slices)
        hist = {k: np.ascontiguousarray(v.numpy()[:500]) for k, v in P.reconstruction_histories(cfg, tr).items()}
        assert len(hist["WEPL"]) == 500
        x0 = (0.95 + 0.1 * np.random.default_rng(3).random(cfg.NUM_VOXELS)).astype(np.float32)
        with Context(cfg) as ctx:
            ctx.set_reconstruction_histories(hist)
            ctx.x_host_2_GPU(x0)
            ctx.DROP_full_tx_iteration(1)
            out.append(ctx.x_GPU_2_host())
    assert np.count_nonzero(np.abs(out[0] - x0) > 1e-5) > 500
    np.testing.assert_allclose(out[0], out[1], rtol=0, atol=2e-6)
