"""Kernels of the training pass at their edges: items of four, two and one rows
of the tensor-core weight gradient, with rows outside the image."""
import numpy as np
import pytest

from test_surrogate import _bf16_bits, _from_bits, _torch

pytestmark = pytest.mark.gpu


# batches large enough for several rows an item (four up to dilation 32, two
# beyond), and one too small for that; heights that leave the last rows of some
# residue classes, or a whole item, outside the image
@pytest.mark.parametrize("shape,dil", [((8, 77, 130), 1), ((8, 77, 130), 5), ((5, 70, 128), 32), ((5, 71, 129), 33),
                                       ((5, 66, 128), 64), ((160, 1, 64), 64), ((40, 5, 65), 4), ((1, 153, 20), 1)])
def test_weight_gradient_rows_per_item(glsu, shape, dil):
    """FP32 sums of exact BF16 products against FP64: a CTA's chain is some
    hundred additions, so errors stay below 100 x 2^-24 of the partial sums and
    those below the largest sum; the biases' chains are compensated."""
    torch = _torch()
    rng = np.random.default_rng(dil)
    B, H, W = shape
    gb = _bf16_bits(rng.uniform(-1, 1, (B, H, W, 32)).astype(np.float32))
    ab = _bf16_bits(rng.uniform(-1, 1, (B, H, W, 32)).astype(np.float32))
    dg, da = (torch.from_numpy(v.view(np.int16)).cuda() for v in (gb, ab))
    dw, db = glsu.wgrad32(dg.data_ptr(), da.data_ptr(), B, W, H, dil)
    again = glsu.wgrad32(dg.data_ptr(), da.data_ptr(), B, W, H, dil)
    assert np.array_equal(dw, again[0]) and np.array_equal(db, again[1])
    g, a = _from_bits(gb).astype(np.float64), _from_bits(ab)
    ap = np.zeros((B, H + 2 * dil, W + 2 * dil, 32))
    ap[:, dil:dil + H, dil:dil + W] = a
    ref = np.zeros((32, 32, 3, 3))
    for ky in range(3):
        for kx in range(3):
            sh = ap[:, ky * dil:ky * dil + H, kx * dil:kx * dil + W]
            ref[:, :, ky, kx] = g.reshape(-1, 32).T @ sh.reshape(-1, 32)
    rdb = g.sum((0, 1, 2))
    assert np.abs(dw - ref).max() <= 1e-5 * np.abs(ref).max()
    assert np.abs(db - rdb).max() <= 1e-6 * np.abs(rdb).max()
