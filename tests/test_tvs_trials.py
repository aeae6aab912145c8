"""Trials of the superiorization accepted in each launch of the chain (4, 4, 8, 16 and the rest), against the
oracle: L exactly, the image to float rounding (the sums of ||G|| are double sums in other orders).

A pure noise image of standard deviation s accepts the first beta = A^L small against s sqrt(voxels); the
amplitudes put that into each launch.  Sizes: a remainder of a block, and more blocks than the grid holds.
"""
import numpy as np
import pytest

from oracle import TvsOracle
from pct_reconstruction_b200 import Config

CASES = [(1.0, 0.9, 1, 4), (0.0055, 0.9, 5, 8), (0.003, 0.9, 9, 16), (0.001, 0.9, 17, 32), (2e-4, 0.9, 33, 134),
         (1e-9, 0.9, 135, 302)]


def config(columns, slices, **extra):
    return Config(COLUMNS=columns, ROWS=columns - 3, SLICES=slices, VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1,
                  RECON_CYL_RADIUS=columns * 0.05, **extra)


def noise(cfg, amplitude):
    rng = np.random.default_rng(5)
    x = (amplitude * np.sqrt(6000.0 / cfg.NUM_VOXELS) * rng.normal(size=cfg.NUM_VOXELS)).astype(np.float32)
    return x, np.ones(cfg.NUM_VOXELS, np.uint8)


@pytest.mark.parametrize("amplitude,A,low,high", CASES)
def test_cases_reach_their_launch(amplitude, A, low, high):
    cfg = config(47, 3, TVS_A=A, TVS_REPETITIONS=1)
    x, hull = noise(cfg, amplitude)
    _, L, _ = TvsOracle(cfg.struct).ntvs_iteration(x, hull, 1, 0)
    assert low <= L <= high


@pytest.mark.gpu
@pytest.mark.parametrize("amplitude,A,low,high", CASES)
@pytest.mark.parametrize("columns,slices", [(47, 3), (170, 9)])
def test_trials_match_oracle(columns, slices, amplitude, A, low, high):
    from pct_reconstruction_b200 import Context
    cfg = config(columns, slices, TVS_A=A)
    x, hull = noise(cfg, amplitude)
    xo, L, _ = TvsOracle(cfg.struct).ntvs_iteration(x, hull, 1, 0)
    with Context(cfg) as ctx:
        ctx.x_host_2_GPU(x)
        ctx.set_array("hull", hull)
        ctx.NTVS_iteration(1)
        assert ctx.tvs_L == L
        np.testing.assert_allclose(ctx.x_GPU_2_host(), xo, rtol=1e-6, atol=1e-7 * max(amplitude, 1e-9))
        assert ctx.counters()["wait_expired"] == 0


@pytest.mark.gpu
def test_image_without_a_variation_to_compare():
    """A NaN in the image: no trial is accepted, the image stays, and each repetition is counted."""
    from pct_reconstruction_b200 import Context
    cfg = config(47, 3, TVS_REPETITIONS=2)
    x, hull = noise(cfg, 0.01)
    x[1234] = np.nan
    with Context(cfg) as ctx:
        ctx.x_host_2_GPU(x)
        ctx.set_array("hull", hull)
        ctx.NTVS_iteration(1)
        np.testing.assert_array_equal(ctx.x_GPU_2_host(), x)
        assert ctx.counters()["wait_expired"] == 2
