"""The table of MLP weights is built with a context's first histories, not with the context; with the first path
layout for histories of the preprocessing."""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import phantoms as P

GRID = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=6.4, SSD_V_SIZE=5.0, MLP_U_STEP=0.05,
            DROP_BLOCK_SIZE=5000, HISTORIES_PER_BLOCK=0, SCATTER_MODE="DETERMINISTIC")


def histories(cfg, n):
    tr = P.simulate_tracks(P.water_cylinder_phantom(6.0), 2 * n, seed=9, continuous_angles=True, t_extent=11.5,
                           v_extent=3.4, span=6.4)
    return {k: v.numpy()[:n] for k, v in P.reconstruction_histories(cfg, tr).items()}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["EXACT", "MIXED"])
def test_table_comes_with_the_first_histories(precision):
    from pct_reconstruction_b200 import Context
    cfg, plain = Config(**GRID, PRECISION=precision), Config(**GRID, PRECISION=precision, EXACT_FAST_POINTS=0)
    h = histories(cfg, 9001)
    x0 = np.full(cfg.NUM_VOXELS, 0.9, np.float32)
    with Context(cfg) as ctx, Context(plain) as none:
        assert ctx.kernel_launches == none.kernel_launches  # the table of steps alone
        for c in (ctx, none):
            c.set_reconstruction_histories(h)
            c.x_host_2_GPU(x0)
        assert ctx.kernel_launches == none.kernel_launches + 1
        assert ctx.path_storage_superblocks == none.path_storage_superblocks == 1
        assert ctx.kernel_launches == none.kernel_launches + 1
        # other histories and a second layout build nothing
        for c in (ctx, none):
            c.set_reconstruction_histories({k: v[1:] for k, v in h.items()})
        launches = ctx.kernel_launches
        ctx.set_path_storage_limit(1 << 30)
        ctx.DROP_full_tx_iteration(1)
        first = ctx.kernel_launches - launches
        launches = none.kernel_launches
        none.set_path_storage_limit(1 << 30)
        none.DROP_full_tx_iteration(1)
        assert none.kernel_launches - launches == first
        if precision == "EXACT":
            np.testing.assert_array_equal(ctx.x_GPU_2_host(), none.x_GPU_2_host())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["EXACT", "MIXED"])
def test_preprocessing_leaves_it_to_the_layout(precision):
    from pct_reconstruction_b200 import Context
    cfg = dict(GRID, T_BIN_SIZE=0.1, V_BIN_SIZE=0.25, ANGULAR_BIN_SIZE=4.0, PRECISION=precision)
    tr = P.simulate_tracks(P.water_cylinder_phantom(6.0), 60000, seed=51, t_extent=13.0, v_extent=3.5)
    td = {k: v.numpy() for k, v in P.tracker_data(tr).items()}
    with Context(Config(**cfg)) as ctx, Context(Config(**cfg, EXACT_FAST_POINTS=0)) as none:
        for c in (ctx, none):
            assert c.preprocessing(td, integer_angles=True) > 10000
        assert ctx.kernel_launches == none.kernel_launches
        before = ctx.mlp_paths()  # the lists of the kernel that an iteration will run
        none.mlp_paths()
        assert ctx.path_storage_superblocks == none.path_storage_superblocks == 1
        assert ctx.kernel_launches == none.kernel_launches + 1
        for a, b in zip(before, ctx.mlp_paths()):
            np.testing.assert_array_equal(a, b)
