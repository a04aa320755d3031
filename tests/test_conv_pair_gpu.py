"""Two convolutions in one call, the first writing the padded input of the second, against the two calls."""
import numpy as np
import pytest
import torch

from glow_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def kernels_of(call):
    """Names of the kernels that a call launches (the nodes of a graph that captures it)."""
    from cuda.bindings import driver
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    handle = driver.CUgraph(graph.raw_cuda_graph())
    _, _, n = driver.cuGraphGetNodes(handle, 0)
    names = []
    for node in driver.cuGraphGetNodes(handle, n)[1]:
        if driver.cuGraphNodeGetType(node)[1] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            err, params = driver.cuGraphKernelNodeGetParams(node)
            assert err == driver.CUresult.CUDA_SUCCESS
            err, name = driver.cuFuncGetName(params.func) if int(params.func) else driver.cuKernelGetName(params.kern)
            assert err == driver.CUresult.CUDA_SUCCESS
            names.append(name.decode())
    return names


# (A second layer of up to 2^19 results and 2^28 products is the few-row kernel's: the pair is two ordinary calls then.)
@pytest.mark.parametrize("n,h,w,cin,mid,oc,k,stride,pad,fused", [
    (4, 33, 31, 64, 64, 80, 3, 1, 1, False),
    (7, 33, 31, 64, 64, 80, 3, 1, 1, True),       # tap pairs
    (3, 40, 29, 128, 128, 64, 3, 1, 1, False),
    (4, 40, 29, 128, 128, 128, 3, 1, 1, True),
    (5, 21, 22, 64, 256, 128, 3, 1, 0, True),     # no padding: no halo
    (6, 27, 26, 256, 128, 128, 3, 2, 1, False),
    (11, 27, 26, 256, 128, 256, 3, 2, 1, True),   # parity planes, odd height
    (9, 14, 15, 256, 256, 512, 3, 2, 1, True),
    (4, 30, 24, 48, 128, 48, 5, 1, 2, True),
    (4, 31, 24, 80, 64, 48, 5, 1, 2, False),
    (6, 31, 24, 80, 64, 48, 5, 1, 2, True),       # an odd last tap of its own in every filter row
    (6, 32, 32, 64, 128, 48, 2, 2, 0, False),
    (30, 32, 32, 64, 128, 96, 2, 2, 0, False),    # a window of which a matrix takes no more room than the planes
    (10, 32, 32, 64, 128, 96, 4, 2, 1, True),     # a window without a centre
    (4, 56, 56, 64, 64, 64, 3, 1, 1, True),       # a block of the image network
    (5, 30, 31, 64, 64, 400, 3, 1, 1, True),      # several column blocks
    (1, 14, 14, 256, 256, 256, 3, 1, 1, False),   # few rows: two ordinary calls
    (2, 40, 40, 32, 96, 32, 3, 1, 1, False),      # neither 64 nor 128 channels
    (2, 40, 40, 32, 72, 32, 3, 1, 1, False),      # rows that are not whole 16-byte pieces
])
@pytest.mark.parametrize("symmetric", [True, False])
def test_pair_equals_the_two_calls(n, h, w, cin, mid, oc, k, stride, pad, fused, symmetric):
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
    layers = [l[0] + l[1:] for l in (first, second)]
    workspace = torch.empty(1 << 26, dtype=torch.uint8, device=DEV)
    names = kernels_of(lambda: ops.channelwise_quantized_conv2d_pair(x, *layers, workspace=workspace))
    main = [k for k in names if "prepare_operands" not in k]   # (that one adds up the first layer's rows)
    assert (len(main) == 2 and all("i8_gemm_requant" in k for k in main)) == fused, names
    forced = second[0] + (second[1], second[2] | ops.FC_FORCE_ANY_SHAPE_KERNEL)
    assert torch.equal(ops.channelwise_quantized_conv2d_pair(x, layers[0], forced), want)
    small = torch.empty(256, dtype=torch.uint8, device=DEV)
    with pytest.raises(Exception, match="workspace"):
        ops.channelwise_quantized_conv2d_pair(x, *layers, workspace=small)
