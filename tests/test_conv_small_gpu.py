"""Convolutions small enough to be one product that reads its windows from the input: the edges of its
row tiles and of its depth steps, taps outside the image, strides, dilations, uneven pads, offsets."""
import numpy as np
import pytest
import torch

from glow_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


CASES = [
    # n, ih, iw, ic, oc, kernel, stride, pads, dilation
    (1, 7, 7, 512, 64, (3, 3), (1, 1), (1, 1, 1, 1), (1, 1)),
    (1, 14, 14, 256, 33, (3, 3), (1, 1), (1, 1, 1, 1), (1, 1)),
    (1, 28, 28, 128, 128, (3, 3), (2, 2), (1, 1, 1, 1), (1, 1)),
    (1, 56, 56, 64, 64, (3, 3), (1, 1), (1, 1, 1, 1), (1, 1)),
    (1, 56, 56, 64, 64, (1, 1), (2, 2), (0, 0, 0, 0), (1, 1)),
    (2, 9, 11, 16, 24, (3, 3), (1, 1), (2, 0, 1, 2), (1, 1)),
    (1, 13, 9, 48, 8, (5, 3), (2, 1), (2, 1, 2, 1), (1, 1)),
    (3, 8, 8, 32, 5, (3, 3), (1, 1), (2, 2, 2, 2), (2, 2)),
    (1, 1, 1, 16, 1, (3, 3), (1, 1), (1, 1, 1, 1), (1, 1)),
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("symmetric", [True, False])
def test_small_convolutions(oracle, case, symmetric):
    n, ih, iw, ic, oc, k, s, p, d = case
    rng = np.random.default_rng(ic + oc)
    K = k[0] * k[1] * ic
    x = rng.integers(-128, 128, (n, ih, iw, ic)).astype(np.int8)
    f = rng.integers(-127, 128, (oc, k[0], k[1], ic)).astype(np.int8)
    bias = rng.integers(-3000, 3000, oc).astype(np.int32)
    fo = np.zeros(oc, np.int32) if symmetric else rng.integers(-3, 4, oc).astype(np.int32)
    bo = np.zeros(oc, np.int32) if symmetric else rng.integers(-5, 5, oc).astype(np.int32)
    fs = rng.uniform(0.002, 0.02, oc).astype(np.float32)
    pp = [t(a) for a in ops.rowwise_requant_params(fs, 0.04, np.float32(0.04) * fs, np.float32(0.9 * np.sqrt(K / 72.0)))]
    status = ops.new_status(DEV)
    args = (t(x), t(f), t(bias), k, s, p, 1, d, -7, 5, t(fo), t(bo), pp[:3], pp[3:], 1, None)
    want = ops.channelwise_quantized_conv2d(*args, flags=ops.FC_FORCE_ANY_SHAPE_KERNEL, status=status)
    got = ops.channelwise_quantized_conv2d(*args, flags=ops.FC_WEIGHT_OFFSETS_ZERO if symmetric else 0, status=status)
    assert torch.equal(got, want) and int(status.item()) == 0
    assert want.numel() < 100 or len(torch.unique(want)) > 10
