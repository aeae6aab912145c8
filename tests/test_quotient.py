"""The backprojection's quotients: the device function against the device's division, and the kernel's two forms
(quotients by reciprocals for a source farther than two radii, divisions for a nearer one) against the oracle."""
import ctypes

import numpy as np
import pytest

from oracle import PreOracle
from pct_reconstruction_b200 import Config, _abi
from pct_reconstruction_b200 import learned as L
from pct_reconstruction_b200 import phantoms as P


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2])
def test_quotient_equals_the_division(seed):
    mismatches = ctypes.c_int64(-1)
    assert _abi.load_library().pct_selftest_quotient(400_000_000, seed, ctypes.byref(mismatches)) == 0
    assert mismatches.value == 0


@pytest.mark.gpu
@pytest.mark.parametrize("source", [1.6, 2.0, 2.01, 30.0])  # in radii
@pytest.mark.parametrize("slices", [1, 6])
def test_backprojection_by_source_distance(source, slices):
    from pct_reconstruction_b200 import Context
    grid = L.scan_config((56, 56, slices), T_BIN_SIZE=0.1, ANGULAR_BIN_SIZE=20.0)
    cfg = Config(**grid, SOURCE_RADIUS=source * grid["RECON_CYL_RADIUS"])
    ph = P.random_ellipsoid_phantom(4, extent=(2.2, 2.0, 0.5 * cfg.RECON_CYL_HEIGHT))
    tr = P.simulate_tracks(ph, 60000, seed=7, device="cuda", continuous_angles=True, t_extent=5.8,
                           v_extent=1.2 * cfg.RECON_CYL_HEIGHT)
    with Context(cfg) as ctx:
        ctx.load_tracker_data(P.tracker_data(tr))
        for st in ("recon_volume_intersections", "binning", "hull_detection", "calculate_means",
                   "sum_squared_deviations", "calculate_standard_deviations", "statistical_cuts", "construct_sinogram", "FBP"):
            ctx.stage(st)
        filtered, fbp = ctx.get_array("sinogram_filtered"), ctx.get_array("FBP_image")
    expected = PreOracle(cfg.struct).backprojection(filtered)
    assert np.count_nonzero(fbp) > 1000
    np.testing.assert_allclose(fbp, expected, rtol=2e-5, atol=1e-4 * max(1.0, np.abs(expected).max()))
