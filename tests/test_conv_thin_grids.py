"""Convolutions on grids one or two voxels high, whose longest patches do not fit in shared memory beside the
weights of 128 input channels: the patch is then a shorter one.

Inputs and weights are small multiples of powers of two whose products and sums are exact in fp32, so the
result has one bf16 rounding: the comparison is exact.
"""
import numpy as np
import pytest

from oracle.unet_oracle import bf16, conv3d

SHAPES = [(2, 1, 200, 128, 16, 0), (1, 2, 126, 128, 128, 0), (3, 1, 54, 128, 32, 0), (2, 2, 100, 128, 64, 1),
          (4, 3, 126, 128, 16, 0), (1, 1, 400, 64, 16, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("nz,ny,nx,cin,cout,up", SHAPES)
def test_convolution_on_thin_grids(nz, ny, nx, cin, cout, up):
    import torch
    from pct_reconstruction_b200.learned import conv3d as gconv
    rng = np.random.default_rng(nz * 1021 + ny * 41 + nx + cin + cout)
    shape = (nz, ny, nx)
    source = tuple(s // 2 for s in shape) if up else shape
    x = rng.integers(-4, 5, source + (cin,)).astype(np.float32)
    w = (rng.integers(-4, 5, (cout, 27, cin)) / 4).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda().to(torch.bfloat16)
    out = gconv(dev(x), cin, shape, dev(w), cout, upsample=up)
    ref = bf16(conv3d(x, w, bool(up)).astype(np.float32))
    np.testing.assert_array_equal(out.float().cpu().numpy().reshape(shape + (cout,)), ref)
