"""The order-independent image update by single voxels and by pairs (196,608 voxels and more), odd counts among
them: the same block sums give the image of the float sums to their rounding, and the same bits each time."""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P


@pytest.mark.gpu
@pytest.mark.parametrize("columns,slices", [(5, 1), (33, 3), (64, 47), (63, 49), (64, 48), (81, 31), (128, 16)])
@pytest.mark.parametrize("precision", ["EXACT", "MIXED"])
def test_update_matches_float_sums(columns, slices, precision):
    from pct_reconstruction_b200 import Context
    R = 0.05 * columns
    p = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=R, COLUMNS=columns, ROWS=columns,
             SLICES=slices, SSD_V_SIZE=slices * 0.25 + 1.0, DROP_BLOCK_SIZE=700, HISTORIES_PER_BLOCK=0, MLP_U_STEP=0.05,
             MIN_MLP_LENGTH=2, LAMBDA=0.01, PRECISION=precision)
    cfg = Config(**p)
    tr = P.simulate_tracks(P.water_cylinder_phantom(0.9 * R), 40000, seed=columns, continuous_angles=True, t_extent=1.8 * R,
                           v_extent=0.8 * cfg.RECON_CYL_HEIGHT, span=R)
    h = {k: v.numpy()[:4001] for k, v in P.reconstruction_histories(cfg, tr).items()}
    x0 = np.linspace(0.8, 1.1, cfg.NUM_VOXELS, dtype=np.float32)
    images = []
    for scatter in ("DETERMINISTIC", "DETERMINISTIC", "ATOMIC"):
        with Context(Config(**p, SCATTER_MODE=scatter)) as ctx:
            ctx.set_reconstruction_histories(h)
            ctx.x_host_2_GPU(x0)
            ctx.DROP_full_tx_iteration(1)
            images.append(ctx.x_GPU_2_host())
    assert np.count_nonzero(images[0] != x0) > min(1000, cfg.NUM_VOXELS // 2)
    np.testing.assert_array_equal(images[0], images[1])
    np.testing.assert_allclose(images[0], images[2], rtol=0, atol=1e-5)  # updates of about 1e-2, float sums of some 1000
