"""The convolution with the residual block's Add in its drain against the two calls it stands for."""
import numpy as np
import pytest
import torch

from glow_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,hw,c,oc,k,add_scale", [
    (2, 40, 64, 256, 1, .7),     # 256-column tiles, a ragged last row tile
    (20, 31, 128, 480, 1, .9),   # 240-column tiles
    (9, 37, 64, 112, 1, .4),     # 128-column tiles, 16 columns short
    (5, 33, 256, 64, 1, 1.3),    # 64-column tiles, taken in turns by half of the warps
    (1, 9, 64, 48, 1, .6),       # few rows
    (2, 12, 128, 64, 3, .6),     # not a plain product: the Add follows
    (2, 20, 64, 72, 1, .6),      # rows that are not whole 16-byte pieces
    (2, 20, 64, 64, 1, .002),    # an Add with a shift before the multiplication
])
@pytest.mark.parametrize("relu,splat", [(0, 5), (1, -128)])
def test_convolution_with_add_equals_the_two_calls(n, hw, c, oc, k, add_scale, relu, splat):
    rng = np.random.default_rng(n * 1000 + hw * 10 + oc)
    to = lambda a: torch.from_numpy(a).to(DEV)
    x, f = to(rng.integers(-128, 128, (n, hw, hw, c), dtype=np.int8)), to(rng.integers(-128, 128, (oc, k, k, c), dtype=np.int8))
    bias, zero = to(rng.integers(-4000, 4000, oc, dtype=np.int32)), torch.zeros(oc, dtype=torch.int32, device=DEV)
    scales = rng.uniform(.002, .02, oc).astype(np.float32)
    pp = [to(a) for a in ops.rowwise_requant_params(scales, .05, np.float32(.05) * scales, .2 * np.sqrt(c * k * k / 64))]
    conv = (x, f, bias, (k, k), (1, 1), (k // 2,) * 4, 1, (1, 1), 3, -7, zero, zero, pp[:3], pp[3:], relu, None)
    other = to(rng.integers(-128, 128, (n, hw, hw, oc), dtype=np.int8))
    add = (-9, 3, 11, ops.quantize_scale_offset_32to8(np.float32(add_scale)), ops.quantize_scale_offset_32to8(np.float32(.8)), splat)
    status = ops.new_status(DEV)
    kw = dict(flags=ops.FC_WEIGHT_OFFSETS_ZERO, status=status)
    lhs = ops.channelwise_quantized_conv2d(*conv, flags=ops.FC_FORCE_ANY_SHAPE_KERNEL)
    assert torch.equal(ops.channelwise_quantized_conv2d(*conv, **kw), lhs)
    a, b = lhs.int(), other.int()

    def side(v, off, t):
        v = (v - off) >> t[0]
        return (v * t[2] + ((1 << t[1]) >> 1)) >> t[1]

    want = (side(a, add[1], add[3]) + side(b, add[2], add[4]) + add[0]).clamp(-128, 127).clamp(min=splat).to(torch.int8)
    assert torch.equal(ops.channelwise_quantized_conv2d_add(*conv, other, *add, **kw), want)
    assert torch.equal(ops.element_add_maxsplat_i8(lhs, other, *add), want)
    assert int(status.item()) == 0 and len(torch.unique(want)) > 20
