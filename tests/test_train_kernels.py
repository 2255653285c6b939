"""Kernels of the training pass at their edges: items of four, two and one rows
of the tensor-core weight gradient, with rows outside the image, and the
backward kernels of the two layers between 2 and 32 channels."""
import numpy as np
import pytest

from oracle import surrogate as S
from test_surrogate import _bf16_bits, _from_bits, _net_case, _torch

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


# heights and widths around the 4-row, 128-pixel items of the first and last
# layer's backward kernels, and dilations that leave whole taps outside
@pytest.mark.parametrize("shape,first,last", [((1, 1, 1), 1, 1), ((1, 5, 3), 2, 64), ((2, 4, 128), 64, 1),
                                              ((2, 9, 129), 1, 3), ((1, 7, 260), 33, 1)])
def test_narrow_layer_gradients(glsu, shape, first, last):
    """Against the oracle with the same BF16 rounding points; what differs is
    FP32 against FP64 sums, and through them a rare BF16 step of one value, as
    in the test of the whole network: 2e-2 of a layer's gradient."""
    dil = [first, 2, 4, 8, 4, 2, 1, last]
    torch, p, z, t = _net_case(glsu, *shape, 11)
    net = glsu.Surrogate(shape[0], shape[2], shape[1], dil, training=True)
    net.params = p
    dz, dt = torch.from_numpy(z).cuda(), torch.from_numpy(t).cuda()
    _, g = net.backward(dz.data_ptr(), dt.data_ptr(), want_grad=True)
    _, again = net.backward(dz.data_ptr(), dt.data_ptr(), want_grad=True)
    net.close()
    assert np.array_equal(g, again)
    _, rg = S.loss_and_grad(p, z.astype(np.complex128), t.astype(np.complex128), dil)
    offs = np.cumsum([0] + [co * ci * 9 + co for co, ci in S.SIZES])
    for k in (0, 6, 7):
        a, b = g[offs[k]:offs[k + 1]].astype(np.float64), rg[offs[k]:offs[k + 1]]
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b)
