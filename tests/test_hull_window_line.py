"""Hull walks on both sides of the line between the two kernels (524,288 histories), against the reference's steps
with every mark in the images directly."""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import learned as L
from test_fast_walks import scan


@pytest.mark.gpu
@pytest.mark.parametrize("n", [524287, 524289])
@pytest.mark.parametrize("columns,slices,discrete", [(64, 8, True), (200, 12, False), (317, 5, False)])
def test_counts_are_identical(n, columns, slices, discrete):
    from pct_reconstruction_b200 import Context
    p = L.scan_config((columns, columns, slices), 60000, 12, SC_UPPER_THRESHOLD=2.0, MSC_LOWER_THRESHOLD=-10.0,
                      MSC_UPPER_THRESHOLD=5.0, SM_LOWER_THRESHOLD=1.0)
    td = {k: v[:n].contiguous() for k, v in scan(Config(**p), n, columns, discrete).items()}
    out = []
    for fast in (1, 0):
        with Context(Config(**p, EXACT_FAST_POINTS=fast)) as ctx:
            assert ctx.load_tracker_data(td, integer_angles=discrete) == n
            for stage in ("recon_volume_intersections", "binning", "hull_detection"):
                ctx.stage(stage)
            out.append({k: ctx.get_array(k) for k in ("SC_hull", "MSC_counts", "SM_counts")})
    a, b = out
    assert (a["SC_hull"] == 0).any() and a["MSC_counts"].max() > 1 and a["SM_counts"].max() > 1
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
