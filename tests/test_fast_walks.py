"""The voxel walks by crossing times (EXACT_FAST_POINTS = 1) against the reference's steps (0).

Hull walks (SC, MSC and SM images) and hull-endpoint walks (kept histories, their end points and first
voxels) have to come out identical: whole numbers and float bits.  The scans cover both grids' shapes,
lines along the axes and diagonals (ties at every step), lines that leave through the top and the
bottom, flat lines, and histories on voxel faces.
"""
import numpy as np
import pytest

from pct_reconstruction_b200 import Config
from pct_reconstruction_b200 import learned as L
from pct_reconstruction_b200 import phantoms as P


def scan(cfg, n, seed, discrete):
    ph = P.random_ellipsoid_phantom(seed, extent=(0.8 * cfg.RECON_CYL_RADIUS, 0.75 * cfg.RECON_CYL_RADIUS,
                                                  0.5 * cfg.RECON_CYL_HEIGHT))
    tr = P.simulate_tracks(ph, n, seed=seed, device="cuda", continuous_angles=not discrete,
                           t_extent=2.1 * cfg.RECON_CYL_RADIUS, v_extent=1.2 * cfg.RECON_CYL_HEIGHT)
    return P.tracker_data(tr)


@pytest.mark.gpu
@pytest.mark.parametrize("columns,slices,discrete,voxel", [(64, 8, False, 0.1), (101, 13, True, 0.1), (160, 24, False, 0.0625)])
def test_preprocessing_is_identical(columns, slices, discrete, voxel):
    from pct_reconstruction_b200 import Context
    R = columns * voxel / 2
    p = L.scan_config((columns, columns, slices), 60000, 12)
    p.update(RECON_CYL_RADIUS=R, VOXEL_WIDTH=voxel, VOXEL_HEIGHT=voxel, COLUMNS=columns, ROWS=columns, SLICES=slices)
    td = scan(Config(**p), 400000, columns, discrete)
    out = []
    for fast in (1, 0):
        with Context(Config(**p, EXACT_FAST_POINTS=fast)) as ctx:
            ctx.load_tracker_data(td, integer_angles=discrete)
            for stage in ("recon_volume_intersections", "binning", "hull_detection"):
                ctx.stage(stage)
            out.append({k: ctx.get_array(k) for k in ("SC_hull", "MSC_counts", "SM_counts")})
            out[-1]["expired"] = ctx.counters()["wait_expired"]
    a, b = out
    assert (a["SC_hull"] == 0).any() and a["MSC_counts"].max() > 1
    assert columns * voxel < 10 or a["SM_counts"].max() > 1  # SM takes water-equivalent lengths from 6 cm on
    for k in ("SC_hull", "MSC_counts", "SM_counts"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert a["expired"] == b["expired"]


def end_points(cfg, n, seed):
    """Entry and exit points on the cylinder with random, axis-parallel and diagonal directions."""
    rng = np.random.default_rng(seed)
    R, H = cfg.RECON_CYL_RADIUS, cfg.RECON_CYL_HEIGHT
    phi = rng.uniform(-np.pi, np.pi, n)
    kind = rng.integers(0, 6, n)
    angle = np.where(kind == 0, rng.uniform(0, 2 * np.pi, n), phi + np.pi + rng.normal(0, 0.5, n))
    angle = np.where(kind == 1, rng.integers(0, 9, n) * (np.pi / 4), angle)      # axes and diagonals
    z = rng.uniform(-0.55 * H, 0.55 * H, n)
    xz = rng.normal(0, 0.02, n)
    xz = np.where(kind == 2, rng.normal(0, 0.6, n), xz)                            # steep
    xz = np.where(kind == 3, 0.0, xz)                                              # flat
    x, y = R * np.cos(phi), R * np.sin(phi)
    on = kind == 4                                                                 # on voxel corners
    x = np.where(on, np.round(x / cfg.VOXEL_WIDTH) * cfg.VOXEL_WIDTH, x)
    y = np.where(on, np.round(y / cfg.VOXEL_HEIGHT) * cfg.VOXEL_HEIGHT, y)
    z = np.where(on, np.round(z / cfg.VOXEL_THICKNESS) * cfg.VOXEL_THICKNESS, z)
    back = rng.permutation(n)
    f = lambda a: a.astype(np.float32)
    return {"x_entry": f(x), "y_entry": f(y), "z_entry": f(z), "x_exit": f(x[back]), "y_exit": f(y[back]),
            "z_exit": f(z[back]), "xy_entry_angle": f(angle), "xz_entry_angle": f(xz),
            "xy_exit_angle": f(angle[back] + np.pi), "xz_exit_angle": f(xz[back]), "WEPL": f(rng.uniform(0, 20, n))}


@pytest.mark.gpu
@pytest.mark.parametrize("columns,slices,n", [(64, 8, 1), (64, 8, 33), (101, 13, 200000), (200, 32, 200000)])
def test_endpoints_are_identical(columns, slices, n):
    from pct_reconstruction_b200 import Context
    p = dict(VOXEL_WIDTH=0.1, VOXEL_HEIGHT=0.1, VOXEL_THICKNESS=0.25, RECON_CYL_RADIUS=columns * 0.05, COLUMNS=columns,
             ROWS=columns, SLICES=slices, SSD_V_SIZE=slices * 0.25 + 1.0)
    cfg = Config(**p)
    hull = P.hull_image(cfg, P.water_cylinder_phantom(0.7 * cfg.RECON_CYL_RADIUS)).numpy().astype(np.uint8)
    hull &= (np.random.default_rng(1).uniform(size=hull.size) < 0.9).astype(np.uint8)  # a porous hull
    h = end_points(cfg, n, columns + n)
    out = []
    for fast in (1, 0):
        with Context(Config(**p, EXACT_FAST_POINTS=fast)) as ctx:
            ctx.set_history_vectors(h)
            ctx.set_array("hull", hull)
            ctx.stage("reconstruction_cuts")
            names = ["first_MLP_voxel_reconstruction"] + [f"{a}_{e}_reconstruction" for a in "xyz" for e in ("entry", "exit")]
            out.append({k: ctx.get_array(k) for k in names} if ctx.reconstruction_histories else {})
    assert out[0].keys() == out[1].keys()
    assert n < 1000 or len(out[0]["x_entry_reconstruction"]) > n // 4
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k].view(np.uint32), out[1][k].view(np.uint32), err_msg=k)


@pytest.mark.gpu
@pytest.mark.parametrize("columns,slices,n", [(64, 8, 530001), (200, 12, 600000), (317, 5, 524288), (330, 4, 524288)])
def test_windowed_counts_are_identical(columns, slices, n):
    """The hull walk's counts in shared memory (524,288 histories or more): all slices in one window, some,
    one with an odd number of voxels, and slices too large for one; histories in one to three of the images.
    Without fast points every mark goes to the images directly."""
    from pct_reconstruction_b200 import Context
    p = L.scan_config((columns, columns, slices), 60000, 12, SC_UPPER_THRESHOLD=2.0, MSC_LOWER_THRESHOLD=-10.0,
                      MSC_UPPER_THRESHOLD=5.0, SM_LOWER_THRESHOLD=1.0)
    td = scan(Config(**p), n, columns, False)
    out = []
    for fast in (1, 0):
        with Context(Config(**p, EXACT_FAST_POINTS=fast)) as ctx:
            ctx.load_tracker_data(td)
            for stage in ("recon_volume_intersections", "binning", "hull_detection"):
                ctx.stage(stage)
            out.append({k: ctx.get_array(k) for k in ("SC_hull", "MSC_counts", "SM_counts")})
    a, b = out
    assert (a["SC_hull"] == 0).any() and a["MSC_counts"].max() > 1 and a["SM_counts"].max() > 1
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
