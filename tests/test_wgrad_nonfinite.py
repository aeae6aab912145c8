"""Weight gradients of inputs with infinities and NaN: they reach the taps that multiply them and no others.

Inputs are small whole numbers, so that every finite sum is exact in fp32 and an infinity gives a signed
infinity or, against a zero of dZ, a NaN; the comparison with float64 sums is exact, NaN included.
"""
import numpy as np
import pytest

# grids with several patches per row, with a patch's last column at each remainder, slices in pairs (16
# input channels) and alone, an upsampled input, and accumulators that are added to dw several times
CASES = [(4, 9, 20, 16, 16, 0), (3, 8, 17, 32, 32, 0), (2, 6, 70, 64, 16, 0), (6, 10, 24, 16, 32, 1),
         (33, 40, 33, 32, 32, 0)]


def reference(x, dz, up):
    """float64 sums over the voxels of dZ, the input's surroundings zero."""
    if up:
        x = x.repeat(2, 0).repeat(2, 1).repeat(2, 2)
    nz, ny, nx, cin = x.shape
    out = np.zeros((dz.shape[3], 27, cin))
    for t in range(27):
        o = (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)
        to, of = zip(*[(slice(max(0, -d), n - max(0, d)), slice(max(0, d), n + min(0, d))) for d, n in zip(o, x.shape)])
        a, b = dz[to].reshape(-1, dz.shape[3]), x[of].reshape(-1, cin)
        # in two parts: 0 x infinity must not depend on how a matrix product is evaluated
        finite = np.isfinite(b)
        out[:, t] = a.T @ np.where(finite, b, 0)
        for v, c in zip(*np.nonzero(~finite)):
            with np.errstate(invalid="ignore"):
                out[:, t, c] += a[v] * b[v, c]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nz,ny,nx,cin,cout,up", CASES)
def test_infinities_reach_only_their_taps(nz, ny, nx, cin, cout, up):
    import torch
    from pct_reconstruction_b200.learned import conv3d_wgrad
    rng = np.random.default_rng(nz * 1031 + ny * 43 + nx + cin + cout)
    shape = (nz, ny, nx)
    source = tuple(s // 2 for s in shape) if up else shape
    x = rng.integers(-3, 4, source + (cin,)).astype(np.float64)
    dz = rng.integers(-3, 4, shape + (cout,)).astype(np.float64)
    # corners, edges of patches (columns 6, 7, 14, 15, 30, 31, rows 1, 2) and anywhere; one channel each
    spots = [(0, 0, 0), tuple(s - 1 for s in source)]
    spots += [(z, y, c) for z in (0, source[0] - 1) for y in (1, 2) for c in (6, 7, 14, 15, 30, 31) if c < source[2]]
    for k, (z, y, c) in enumerate(spots):
        x[z, y, c, k % cin] = (np.inf, -np.inf, np.nan)[k % 3]
    dev = lambda a: torch.from_numpy(a.astype(np.float32)).cuda().to(torch.bfloat16)
    got = conv3d_wgrad(dev(x), cin, shape, dev(dz), cout, upsample=up).cpu().numpy().reshape(cout, 27, cin)
    np.testing.assert_array_equal(got, reference(x, dz, up).astype(np.float32))
