"""Two convolutions in one call, the first writing the padded input of the second, against the two calls."""
import numpy as np
import pytest
import torch

from glow_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,h,w,cin,mid,oc,k,stride,pad", [
    (4, 33, 31, 64, 64, 80, 3, 1, 1),      # tap pairs
    (3, 40, 29, 128, 128, 64, 3, 1, 1),
    (5, 21, 22, 64, 256, 128, 3, 1, 0),    # no padding: no halo
    (6, 27, 26, 256, 128, 128, 3, 2, 1),   # parity planes, odd height
    (9, 14, 15, 256, 256, 512, 3, 2, 1),
    (4, 30, 24, 48, 128, 48, 5, 1, 2),
    (4, 31, 24, 80, 64, 48, 5, 1, 2),      # an odd last tap of its own in every filter row
    (6, 32, 32, 64, 128, 48, 2, 2, 0),     # a window without a centre
    (1, 14, 14, 256, 256, 256, 3, 1, 1),   # few rows: two ordinary calls
    (2, 40, 40, 32, 96, 32, 3, 1, 1),      # neither 64 nor 128 channels
    (2, 40, 40, 32, 72, 32, 3, 1, 1),      # rows that are not whole 16-byte pieces
])
@pytest.mark.parametrize("symmetric", [True, False])
def test_pair_equals_the_two_calls(n, h, w, cin, mid, oc, k, stride, pad, symmetric):
    rng = np.random.default_rng(h * 100 + mid)
    to = lambda a: torch.from_numpy(a).to(DEV)
    x = to(rng.integers(-128, 128, (n, h, w, cin), dtype=np.int8))

    def layer(ci, co, k, stride, pad, out_off, in_off, relu, zero):
        f = to(rng.integers(-128, 128, (co, k, k, ci), dtype=np.int8))
        scales = rng.uniform(.002, .02, co).astype(np.float32)
        pp = [to(a) for a in ops.rowwise_requant_params(scales, .05, np.float32(.05) * scales, .2 * np.sqrt(ci * k * k / 64))]
        offsets = to(np.zeros(co, np.int32) if zero else rng.integers(-9, 9, co, dtype=np.int32))
        args = (f, to(rng.integers(-4000, 4000, co, dtype=np.int32)), (k, k), (stride, stride), (pad,) * 4, 1, (1, 1), out_off, in_off,
                offsets, torch.zeros(co, dtype=torch.int32, device=DEV), pp[:3], pp[3:], relu, None)
        return args, ops.i8_row_sums(f.view(co, -1)), ops.FC_WEIGHT_OFFSETS_ZERO if zero else 0

    first, second = layer(cin, mid, 1, 1, 0, -20, 5, 1, symmetric), layer(mid, oc, k, stride, pad, 7, -20, 0, True)
    between = ops.channelwise_quantized_conv2d(x, *first[0], flags=first[2])
    want = ops.channelwise_quantized_conv2d(between, *second[0], flags=second[2])
    status = ops.new_status(DEV)
    for sums in (True, False):   # the filters' row sums are the caller's, or are worked out
        layers = [l[0] + (l[1] if sums else None, l[2]) for l in (first, second)]
        got = ops.channelwise_quantized_conv2d_pair(x, *layers, status=status)
        assert torch.equal(got, want)
    assert int(status.item()) == 0 and len(torch.unique(want)) > 20
    small = torch.empty(256, dtype=torch.uint8, device=DEV)
    with pytest.raises(Exception, match="workspace"):
        ops.channelwise_quantized_conv2d_pair(x, *layers, workspace=small)
