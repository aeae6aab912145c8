"""End points on grids of few slices, whose lines leave through the top after a few steps: warps with such lines
take the reference's steps, and the others go by crossing times.  Both, and the kernel without crossing times,
give the same end points, first voxels and histories."""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P
from test_fast_walks import end_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns,slices", [(48, 1), (200, 1), (200, 2), (200, 4), (200, 16), (200, 17), (316, 1)])
@pytest.mark.parametrize("steep", [False, True])
def test_endpoints_are_identical(columns, slices, steep):
    from pct_reconstruction_b200 import Context
    p = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=columns * 0.05, COLUMNS=columns,
             ROWS=columns, SLICES=slices, SSD_V_SIZE=slices * 0.25 + 1.0)
    cfg = Config(**p)
    hull = P.hull_image(cfg, P.water_cylinder_phantom(0.7 * cfg.RECON_CYL_RADIUS)).numpy().astype(np.uint8)
    hull &= (np.random.default_rng(1).uniform(size=hull.size) < 0.9).astype(np.uint8)
    h = end_points(cfg, 150_001, columns + slices)
    if not steep:  # a scan's elevations: some warps without a line that leaves early
        for e in ("xz_entry_angle", "xz_exit_angle"):
            h[e] = (0.02 * cfg.RECON_CYL_HEIGHT / cfg.RECON_CYL_RADIUS * np.random.default_rng(2).normal(size=len(h[e]))).astype(np.float32)
    out = []
    for fast in (1, 0):
        with Context(Config(**p, EXACT_FAST_POINTS=fast)) as ctx:
            ctx.set_history_vectors(h)
            ctx.set_array("hull", hull)
            ctx.stage("reconstruction_cuts")
            names = ["first_MLP_voxel_reconstruction"] + [f"{a}_{e}_reconstruction" for a in "xyz" for e in ("entry", "exit")]
            out.append({k: ctx.get_array(k) for k in names})
    assert len(out[0]["x_entry_reconstruction"]) > 10_000
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k].view(np.uint32), out[1][k].view(np.uint32), err_msg=k)
