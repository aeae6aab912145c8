"""An unconditioned perturbation of an image with an infinity: ||G|| is NaN and so is the direction in every
hull voxel, those of flat regions (G = 0) among them; outside the hull the image stays.  A NaN voxel by itself
compares false in |grad| > 0 and reaches nothing."""
import numpy as np
import pytest

from oracle import TvsOracle
from pct_reconstruction_b200 import Config


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, -np.inf, 3e38, np.nan])
def test_nonfinite_voxel_matches_oracle(value):
    from pct_reconstruction_b200 import Context
    cfg = Config(COLUMNS=47, ROWS=44, SLICES=3, VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, RECON_CYL_RADIUS=2.35,
                 TVS_CONDITIONED=0, TVS_REPETITIONS=2)
    x = np.zeros(cfg.NUM_VOXELS, np.float32)
    x[500:900] = 1
    x[1234] = value
    hull = np.ones(cfg.NUM_VOXELS, np.uint8)
    hull[3000:] = 0
    xo, L, _ = TvsOracle(cfg.struct).ntvs_iteration(x, hull, 1, 0)
    with Context(cfg) as ctx:
        ctx.x_host_2_GPU(x)
        ctx.set_array("hull", hull)
        ctx.NTVS_iteration(1)
        assert ctx.tvs_L == L
        np.testing.assert_allclose(ctx.x_GPU_2_host(), xo, rtol=1e-6, atol=1e-7)
