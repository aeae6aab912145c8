"""Filter, backprojection and median filter at the edges of their tiles, against the oracle.

Bins: more detector bins than one tile of the filter (256) and fewer than one of its CTAs (128), angle
bins and slices that leave a remainder of the strips (6) and slice groups (8).  Median: the radii with
their own network (1, 2, 3) and one without (4); a sparse scan leaves medians of exactly zero, which
are selected by counting.  Tolerances: every term is rounded to float as the oracle rounds it, so sums
differ by the library functions' last places (the tolerance of the head-size comparison); medians of
the same image are the same value.
"""
from fractions import Fraction

import numpy as np
import pytest

from oracle import PreOracle
from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import learned as L
from pct_reconstruction_b200 import phantoms as P


@pytest.mark.gpu
@pytest.mark.parametrize("columns,slices,t_size,angle,filter_type,radius,n", [
    (64, 8, 0.25, 12.0, 1, 3, 200000),   # fewer bins than one CTA, 30 strips
    (101, 13, 0.035, 8.0, 0, 1, 300000),  # more than one tile, 45 angles, 13 slices
    (64, 1, 0.1, 360.0, 2, 2, 2000),     # one angle, one slice, unfiltered, sparse
    (48, 17, 0.1, 36.0, 0, 4, 3000),     # sparse, radius without a network
    (48, 9, 0.1, 36.0, 1, 3, 3000)])     # sparse
def test_filter_backprojection_median(columns, slices, t_size, angle, filter_type, radius, n):
    from pct_reconstruction_b200 import Context
    cfg = Config(**L.scan_config((columns, columns, slices), T_BIN_SIZE=t_size, ANGULAR_BIN_SIZE=angle,
                                 SINOGRAM_FILTER=filter_type, FBP_MED_FILTER_RADIUS=radius))
    R = cfg.RECON_CYL_RADIUS
    ph = P.random_ellipsoid_phantom(3, extent=(0.8 * R, 0.75 * R, 0.5 * cfg.RECON_CYL_HEIGHT))
    tr = P.simulate_tracks(ph, n, seed=columns, device="cuda", continuous_angles=True, t_extent=2.1 * R,
                           v_extent=1.2 * cfg.RECON_CYL_HEIGHT)
    o = PreOracle(cfg.struct)
    with Context(cfg) as ctx:
        ctx.load_tracker_data(P.tracker_data(tr))
        for st in ("recon_volume_intersections", "binning", "hull_detection", "calculate_means",
                   "sum_squared_deviations", "calculate_standard_deviations", "statistical_cuts"):
            ctx.stage(st)
        sums, counts = ctx.get_array("sinogram"), ctx.get_array("bin_counts")
        ctx.stage("construct_sinogram")
        ctx.stage("FBP")
        filtered, fbp, med = (ctx.get_array(k) for k in ("sinogram_filtered", "FBP_image", "FBP_median_filtered"))
    assert np.count_nonzero(sums) > 0
    _, o_filtered = o.sinogram_filter(counts, sums)
    np.testing.assert_allclose(filtered, o_filtered, rtol=2e-5, atol=1e-4)
    np.testing.assert_allclose(fbp, o.backprojection(filtered), rtol=2e-5, atol=1e-4)
    np.testing.assert_array_equal(med, o.median_filter(fbp, radius))


def test_quotient_is_correctly_rounded():
    """The backprojection's quotients by a reciprocal: two residual corrections, in exact arithmetic."""
    def fma(a, b, c):
        return float(Fraction(a) * Fraction(b) + Fraction(c))

    rng = np.random.default_rng(0)
    for i in range(6000):
        source = rng.uniform(20, 400)
        b = source + rng.uniform(-0.5, 0.5) * source
        a = rng.uniform(-20, 20)
        if i % 3 == 0:  # mantissas of ones
            b = float(np.nextafter(2.0 ** rng.integers(3, 9), 0))
        if i % 3 == 1:  # bin sizes and voxel positions
            a, b = float(rng.integers(-200, 200)) * 0.125, float(rng.integers(1, 1000)) * 0.05
        r = float(Fraction(1) / Fraction(b))
        q = a * r
        for _ in range(2):
            q = fma(fma(-q, b, a), r, q)
        assert q == a / b
