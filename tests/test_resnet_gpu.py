"""ResNet-50 v1.5 int8 on the GPU against the same quantized network on the CPU oracle: every
layer is integer arithmetic, so the int8 logits must match bit for bit."""
import numpy as np
import pytest
import torch

from glow_b200 import ops, resnet

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run_oracle(oracle, layers, q, x_nchw):
    """The same quantized network through the CPU oracle (numpy in, int8 logits out)."""
    tqp = q["tqp"]
    x = oracle.element_quantize_i8(np.ascontiguousarray(np.transpose(x_nchw, (0, 2, 3, 1))), *tqp["input"])

    def conv(name, t):
        c = q["conv"][name]
        spec = c["spec"]
        k, s, p = (spec["k"],) * 2, (spec["stride"],) * 2, (spec["pad"],) * 4
        ohw = ops.conv_out_hw(t.shape[1:3], k, s, p)
        return oracle.conv2d_i8_i32(t, c["filter"], c["bias"], ohw, k, s, p, 1, (1, 1), c["out_offset"], c["in_offset"],
                                    c["filter_offsets"], c["bias_offsets"], c["params"][:3], c["params"][3:],
                                    1 if spec["relu"] else 0, None)

    for l in layers:
        if l[0] == "conv":
            x = conv(l[1]["name"], x)
        elif l[0] == "maxpool":
            x = oracle.max_pool_i8(x, ops.conv_out_hw(x.shape[1:3], (3, 3), (2, 2), (1, 1, 1, 1)), (3, 3), (2, 2), (1, 1, 1, 1),
                                   tqp["conv1"][1])
        elif l[0] == "block":
            y = x
            for c in l[2]:
                y = conv(c["name"], y)
            sc = conv(l[3]["name"], x) if l[3] else x
            a = q["add"][l[1]]
            out_off = tqp[a["out"]][1]
            x = oracle.element_add_i8(y, sc, out_off, tqp[a["lhs"]][1], tqp[a["rhs"]][1], a["lhs_triple"], a["rhs_triple"])
            x = oracle.element_maxsplat_i8(x, out_off)
        elif l[0] == "avgpool":
            src = q["avgpool_in"]
            hw = x.shape[1]
            tr = ops.quantize_scale_offset_32to8(np.float32(tqp[src][0]) / np.float32(tqp["avgpool"][0]) / np.float32(hw * hw))
            x = oracle.avg_pool_i8(x, (1, 1), (hw, hw), (1, 1), (0, 0, 0, 0), True, tqp["avgpool"][1], tqp[src][1], tr)
        elif l[0] == "fc":
            f = q["fc"]
            x = oracle.rowwise_quantized_fc_i8_i32(x.reshape(x.shape[0], -1), f["w"], f["bias"], f["w_offsets"], f["params"][:3],
                                                   f["params"][3:], tqp["fc"][1], tqp[f["in_name"]][1], 0)
    return x


@pytest.fixture(scope="module")
def net():
    layers = resnet.architecture(num_classes=100)
    w = resnet.float_weights(layers)
    g = torch.Generator().manual_seed(7)
    calib = torch.randn((4, 3, 64, 64), generator=g)
    _, ranges = resnet.float_forward(layers, w, calib, DEV)
    q = resnet.quantize_network(layers, w, ranges)
    return layers, w, q


def test_resnet50_int8_bit_exact_against_oracle(oracle, net):
    layers, w, q = net
    model = resnet.ResNet50Int8(layers, q, DEV)
    g = torch.Generator().manual_seed(11)
    x = torch.randn((2, 3, 64, 64), generator=g)
    logits = model.forward(x.to(DEV))
    torch.cuda.synchronize()
    assert int(model.status.item()) == 0
    want = run_oracle(oracle, layers, q, x.numpy())
    np.testing.assert_array_equal(model.logits_q.cpu().numpy(), want)
    assert len(np.unique(want)) > 20
    # and the quantized network still tracks the fp32 one (quantisation error only)
    ref, _ = resnet.float_forward(layers, w, x, DEV)
    err = (logits - ref).abs().max() / (ref.max() - ref.min())
    assert float(err) < 0.25
    assert model.launches > 100


def test_every_conv_takes_the_tensor_core_path(net):
    """All 53 convolutions of the network are group-1 and land on the contraction kernel
    (im2col or direct); their results equal the direct kernel's on a real activation."""
    layers, w, q = net
    rng = np.random.default_rng(3)
    for name in ("conv1", "s1b0_b", "s2b0_b", "s3b0_b", "s2b0_sc", "s4b2_c"):
        c = q["conv"][name]
        spec = c["spec"]
        x = torch.from_numpy(rng.integers(-128, 128, (2, 20, 20, spec["cin"]), dtype=np.int8)).to(DEV)
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
        pp = [to(a) for a in c["params"]]
        args = (x, to(c["filter"]), to(c["bias"]), (spec["k"],) * 2, (spec["stride"],) * 2, (spec["pad"],) * 4, 1, (1, 1),
                c["out_offset"], c["in_offset"], to(c["filter_offsets"]), to(c["bias_offsets"]), pp[:3], pp[3:],
                1 if spec["relu"] else 0, None)
        assert not c["filter_offsets"].any()  # symmetric filters
        a = ops.channelwise_quantized_conv2d(*args, flags=ops.FC_WEIGHT_OFFSETS_ZERO)
        b = ops.channelwise_quantized_conv2d(*args, flags=ops.FC_FORCE_ANY_SHAPE_KERNEL)
        assert torch.equal(a, b)



def test_programmatic_launches_do_not_change_results(net):
    """The library's kernels start beside their predecessors' tails (programmatic dependent launch)
    and touch global memory only after them: the whole network gives the same bytes with the
    switch off, on, and replayed from a CUDA graph captured with it on."""
    layers, w, q = net
    model = resnet.ResNet50Int8(layers, q, DEV)
    x = torch.randn((3, 3, 96, 96), generator=torch.Generator().manual_seed(5)).to(DEV)
    with ops.programmatic_launch(False):
        model.forward(x)
        plain = model.logits_q.clone()
    with ops.programmatic_launch(True):
        for _ in range(3):
            model.forward(x)
            assert torch.equal(model.logits_q, plain)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            model.forward(x)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                model.forward(x)
                captured = model.logits_q
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, plain)
    assert int(model.status.item()) == 0


@pytest.mark.parametrize("shapes", [((1, 3, 64, 64),) * 4, ((2, 3, 64, 64), (3, 3, 96, 96), (3, 3, 96, 96), (2, 3, 64, 64), (2, 3, 64, 64))])
def test_replayed_forward_equals_the_launches(net, shapes):
    """From the second call of a shape on the layers are replayed from a graph: other images, other
    streams and other shapes in between give what the launches give, and results stay the caller's."""
    layers, w, q = net
    model, plain = resnet.ResNet50Int8(layers, q, DEV), resnet.ResNet50Int8(layers, q, DEV)
    plain.REPLAY_PIXELS = 0
    g = torch.Generator(device=DEV).manual_seed(9)
    xs = [torch.randn(s, device=DEV, generator=g) for s in shapes]
    want = [plain.forward(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got, quantized = [], []
    for x, s in zip(xs, streams):
        with torch.cuda.stream(s):
            got.append(model.forward(x))
            quantized.append(model.logits_q)
    torch.cuda.synchronize()
    assert model.launches == plain.launches and int(model.status.item()) == 0
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert len({t.data_ptr() for t in quantized}) == len(xs)


def test_alternating_shapes_are_captured_once(net):
    """Shapes that take turns are replayed, each from its own graph; more of them than are kept run launch by launch;
    calls on several streams wait for one another."""
    layers, w, q = net
    model, plain = resnet.ResNet50Int8(layers, q, DEV), resnet.ResNet50Int8(layers, q, DEV)
    plain.REPLAY_PIXELS = 0
    captures, capture = [], model._capture
    model._capture = lambda shape: captures.append(shape) or capture(shape)
    g = torch.Generator(device=DEV).manual_seed(2)
    xs = [torch.randn((n, 3, 64, 64), device=DEV, generator=g) for n in (1, 2, 3, 4, 5, 6)]
    want = [plain.forward(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got, call = [], 0
    for turn in range(12):
        for i in ((0, 1, 2) if turn < 6 else range(6)):
            with torch.cuda.stream(streams[call % 3]):
                got.append((i, model.forward(xs[i])))
            call += 1
    torch.cuda.synchronize()
    assert int(model.status.item()) == 0 and all(torch.equal(out, want[i]) for i, out in got)
    assert len(captures) == resnet.Replays.KEPT and len(set(captures)) == len(captures)


@pytest.mark.parametrize("replayed", [False, True])
def test_a_call_on_another_stream_waits_for_the_last(net, replayed):
    """The calls of a model share its workspace and buffers: one on a second stream does not start before the first
    one, still queued behind other work of its stream, has ended."""
    layers, w, q = net
    model = resnet.ResNet50Int8(layers, q, DEV)
    if not replayed:
        model.REPLAY_PIXELS = 0
    g = torch.Generator(device=DEV).manual_seed(8)
    xs = [torch.randn((n, 3, 64, 64), device=DEV, generator=g) for n in (3, 2, 1)]
    want = [[model.forward(x) for _ in range(3)][-1] for x in xs]   # (captured by now, each shape a graph)
    streams, ended, got = [torch.cuda.Stream() for _ in xs], [torch.cuda.Event() for _ in xs], []
    torch.cuda.synchronize()
    for x, s, e in zip(xs, streams, ended):
        with torch.cuda.stream(s):
            if x is xs[0]:
                torch.cuda._sleep(100_000_000)   # some 50 ms
            got.append(model.forward(x))
            e.record()
    streams[-1].synchronize()
    assert all(e.query() for e in ended)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_a_captured_forward_outlives_larger_calls(net):
    """A graph that a caller captured addresses the workspace of that time: it stays when a later call needs more."""
    layers, w, q = net
    model = resnet.ResNet50Int8(layers, q, DEV)
    g = torch.Generator(device=DEV).manual_seed(4)
    x = torch.randn((1, 3, 64, 64), device=DEV, generator=g)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = model.forward(x).clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = model.forward(x)
        small = model.ws
        model.forward(torch.randn((6, 3, 128, 128), device=DEV, generator=g))
        assert model.ws is not small and any(t is small for t in model._captured)
        address = small.data_ptr()
        del small
        fill = [torch.full((1 << 20,), 85, dtype=torch.uint8, device=DEV) for _ in range(64)]
        assert all(not f.data_ptr() <= address < f.data_ptr() + f.numel() for f in fill)
        graph.replay()
        torch.cuda.synchronize()
    assert torch.equal(out, want) and int(model.status.item()) == 0
