"""Weight gradients on the tensor cores (k_wgrad.cu) against whole-number sums.

Inputs are whole numbers from -3 to 3, so every product and every sum is exact in FP32 in
any order (at most 9 times 16384 pixels) and the partials must add up to the whole-number
result exactly: every layer's channels, views into wider tensors, the padded three input
channels, images at the sizes where the tiles change (rows of 8 to 256 pixels, several rows
a tile), borders, one split, several and a last one that is shorter.
"""
import numpy as np
import pytest

from tests import kernel_entries

pytestmark = pytest.mark.gpu


def bf16(a):
    return (a.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)


# input channels, of a tensor with, from, output channels
LAYERS = [(3, 16, 0, 32), (32, 32, 0, 32), (32, 96, 64, 64), (64, 64, 0, 64), (64, 192, 128, 128), (128, 128, 0, 128),
          (128, 256, 128, 128), (256, 256, 0, 128), (192, 192, 0, 64), (96, 96, 0, 32)]


@pytest.mark.parametrize("cin,x_tot,x_off,cout", LAYERS)
@pytest.mark.parametrize("nb,H,W", [(1, 8, 8), (3, 16, 16), (1, 6, 64), (2, 20, 128), (1, 33, 256), (1, 128, 128)])
def test_partials_add_up_exactly(gpu_lib, cin, x_tot, x_off, cout, nb, H, W):
    L = kernel_entries.load()
    rng = np.random.default_rng(cin + x_off + cout + W + H)
    x = rng.integers(-3, 4, (nb, H, W, x_tot))
    if cin == 3:
        x[..., 3:] = 0
    dz = rng.integers(-3, 4, (nb, H, W, cout))
    splits = L.entry_wgrad_splits(nb, H, W, cin)
    part = np.full((splits, cout, 9, cin), np.nan, np.float32)
    P = kernel_entries.ptr
    xb, zb = np.ascontiguousarray(bf16(x)), np.ascontiguousarray(bf16(dz))
    assert L.entry_wgrad(P(xb), x_tot, x_off, cin, P(zb), cout, nb, H, W, P(part)) == 0
    assert np.all(np.isfinite(part))
    xp = np.zeros((nb, H + 2, W + 2, cin))
    xp[:, 1:-1, 1:-1] = x[..., x_off:x_off + cin]
    z = dz.reshape(-1, cout).astype(np.float64)
    want = np.stack([z.T @ xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, cin) for t in range(9)], axis=1)
    assert np.abs(want).max() < 2 ** 24
    assert np.array_equal(part.astype(np.float64).sum(axis=0), want)
