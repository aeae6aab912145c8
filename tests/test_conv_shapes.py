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


# the weight gradient's patches are W x 2 voxels, W = 7, 15, ..., 63; slices in pairs for 16 input channels;
# accumulators are added to dw after at most 96 steps of 16 positions (the last two shapes: several times)
WGRAD_SHAPES = [(1, 1, 1, 16, 16, 0), (2, 1, 8, 16, 32, 0), (3, 5, 63, 16, 16, 0), (5, 2, 64, 16, 128, 0),
                (1, 3, 9, 32, 16, 0), (2, 2, 2, 32, 32, 1), (7, 9, 31, 64, 64, 0), (4, 6, 30, 128, 32, 1),
                (4, 25, 25, 128, 128, 0), (33, 60, 70, 16, 16, 0), (40, 60, 58, 64, 32, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("nz,ny,nx,cin,cout,up", WGRAD_SHAPES)
def test_weight_gradient_is_exact_on_exact_inputs(nz, ny, nx, cin, cout, up):
    import torch
    from oracle.unet_oracle import conv3d_wgrad
    from pct_reconstruction_b200.learned import conv3d_wgrad as gwgrad
    rng = np.random.default_rng(nz * 1013 + ny * 37 + nx + cin + cout)
    shape = (nz, ny, nx)
    source = tuple(s // 2 for s in shape) if up else shape
    x = rng.integers(-3, 4, source + (cin,)).astype(np.float32)   # |sum| <= 9 * 139,200 < 2^24
    dz = rng.integers(-3, 4, shape + (cout,)).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda().to(torch.bfloat16)
    got = gwgrad(dev(x), cin, shape, dev(dz), cout, upsample=up).cpu().numpy()
    np.testing.assert_array_equal(got, conv3d_wgrad(x, dz, bool(up)).astype(np.float32).reshape(-1))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 8, 8), (16, 40, 24)])
def test_bias_gradients_are_the_sums_of_the_layer_gradients(shape):
    """The bias gradient of the output layer is the sum of the loss gradient, 2 (y - t) / count over the hull
    in bf16, which an untrained network (y = x_0) lets the test form itself."""
    import torch
    from oracle.unet_oracle import param_layout
    from pct_reconstruction_b200.learned import UNet
    rng = np.random.default_rng(3)
    v = int(np.prod(shape))
    x0 = rng.uniform(0.5, 1.5, v).astype(np.float32)
    target = (x0 + rng.normal(0, 0.1, v)).astype(np.float32)
    hull = (rng.uniform(size=v) < 0.7).astype(np.uint8)
    T = [torch.from_numpy(a).cuda() for a in (x0, hull, target)]
    with UNet(shape[2], shape[1], shape[0], seed=2) as net:
        _, g = net.gradients(*T)
    d = np.where(hull, x0 - target, 0).astype(np.float64)
    expected = bf16((2 * d / hull.sum()).astype(np.float32)).astype(np.float64)
    got = g[param_layout()[0][-1][1]:]
    assert abs(got[0] - expected.sum()) <= 1e-6 * np.abs(expected).sum()
    assert not got[1:].any()


@pytest.mark.gpu
def test_convolutions_from_many_threads():
    """More calls at once than there are status words, each on its own stream, next to one another."""
    import threading

    import torch
    from pct_reconstruction_b200.learned import conv3d as gconv
    rng = np.random.default_rng(8)
    shape = (6, 20, 30)
    x = torch.from_numpy(rng.integers(-4, 5, shape + (16,)).astype(np.float32)).cuda().to(torch.bfloat16)
    w = torch.from_numpy((rng.integers(-4, 5, (16, 27, 16)) / 4).astype(np.float32)).cuda().to(torch.bfloat16)
    expected = gconv(x, 16, shape, w, 16)
    torch.cuda.synchronize()
    wrong = []

    def work():
        stream = torch.cuda.Stream()
        for _ in range(5):
            with torch.cuda.stream(stream):
                out = gconv(x, 16, shape, w, 16, stream=stream)
                if not torch.equal(out, expected):
                    wrong.append(1)

    threads = [threading.Thread(target=work) for _ in range(80)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
