"""The slab convolution at the edges of its tiling, against the oracle's convolution.

Patches are W x H voxels with (W + 2) (H - 1) + W <= 128, runs of slices are powers of two or the whole
grid, and a CTA goes on with further tiles: grids of one voxel, one row, one column and one slice, grids
one more than a patch, upsampled inputs, and a grid with several tiles per CTA.  Inputs and weights are
small multiples of powers of two whose products and sums are exact in fp32, so the result has one bf16
rounding: the comparison is exact.
"""
import numpy as np
import pytest

from oracle.unet_oracle import bf16, conv3d

SHAPES = [(1, 1, 1, 16, 16, 0), (1, 1, 130, 16, 16, 0), (1, 131, 1, 16, 32, 0), (5, 1, 1, 32, 16, 0),
          (2, 4, 62, 16, 16, 1), (2, 10, 12, 128, 128, 1), (3, 11, 11, 64, 16, 0), (33, 3, 7, 16, 64, 0),
          (7, 13, 31, 32, 64, 0), (4, 25, 25, 128, 16, 0), (18, 8, 26, 16, 128, 1), (40, 60, 59, 16, 16, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("nz,ny,nx,cin,cout,up", SHAPES)
def test_convolution_is_exact_on_exact_inputs(nz, ny, nx, cin, cout, up):
    import torch
    from pct_reconstruction_b200.learned import conv3d as gconv
    rng = np.random.default_rng(nz * 1009 + ny * 31 + nx + cin + cout)
    shape = (nz, ny, nx)
    source = tuple(s // 2 for s in shape) if up else shape
    x = rng.integers(-4, 5, source + (cin,)).astype(np.float32)      # |sum| < 27 * 128 * 16 = 2^16 at most
    w = (rng.integers(-4, 5, (cout, 27, cin)) / 4).astype(np.float32)
    b = rng.integers(-8, 9, cout).astype(np.float32)
    r = rng.integers(-8, 9, shape + (cout,)).astype(np.float32)
    m = rng.integers(-2, 3, shape + (cout,)).astype(np.float32)
    ref = conv3d(x, w, bool(up)).astype(np.float32) + b + r
    ref = bf16(np.where(m > 0, np.maximum(ref, 0), 0))
    dev = lambda a: torch.from_numpy(a).cuda().to(torch.bfloat16)
    out = gconv(dev(x), cin, shape, dev(w), cout, upsample=up, bias=torch.from_numpy(b).cuda(), residual=dev(r),
                mask=dev(m), relu=True)
    np.testing.assert_array_equal(out.float().cpu().numpy().reshape(shape + (cout,)), ref)
