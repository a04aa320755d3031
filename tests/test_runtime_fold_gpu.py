"""What compile() does for a recommendation model's graph: InsertTensor copies of pooled vectors folded
into the pooling launch, a Splat of weights done once, the list replayed as a graph -- and the cases in
which it must keep its hands off.  Results are compared with the same network built so that nothing folds."""
import numpy as np
import pytest

from glow_b200 import ops, runtime, workloads

pytestmark = pytest.mark.gpu
B, D, ROWS, T, CAP = 5, 16, 200, 3, 64


@pytest.fixture()
def dm():
    d = runtime.DeviceManager(0).init()
    yield d
    d.stop()


def network(name, tables, variant):
    f = runtime.Function(name)
    idx, ln = f.placeholder("idx", T * CAP * 4), f.placeholder("len", T * B * 4)
    out, extra = f.placeholder("out", B * (T * D + 8) * 4), f.placeholder("extra", B * D * 4)
    ones, mid = f.activation("ones", CAP * 4), f.activation("mid", T * B * D * 4)
    f.splat(ones, n=CAP, value=1.0)
    if variant == "splat_written":        # not a constant: the weights change between the tables
        f.splat((ones, 0), n=CAP // 2, value=0.5)
    pools = lambda t: f.frwq_slws((mid, t * B * D * 4), f.constant("t%d" % t, tables[t]), ones, (idx, t * CAP * 4),
                                  (ln, t * B * 4), kind=ops.UINT8_FUSED, rows=ROWS, in_line=D + 8, out_line=D, segments=B,
                                  num_indices=CAP, idx64=False)
    insert = lambda t, column: f.insert_tensor(out, (mid, t * B * D * 4), rows=B, width_bytes=D * 4,
                                               dest_pitch_bytes=(T * D + 8) * 4, dest_offset_bytes=column * 4)
    for t in range(T):
        pools(t)
    if variant == "read_elsewhere":       # the pooled vectors of table 1 have another reader
        f.copy(extra, (mid, B * D * 4), nbytes=B * D * 4)
    for t in range(T):
        insert(t, t * D + (0 if variant != "overlapping" else -8 * t))
    if variant == "twice":                # ... and those of table 0 go to two places
        insert(0, T * D - 8)
    return f.compile()


@pytest.mark.parametrize("variant", ["plain", "splat_written", "read_elsewhere", "overlapping", "twice"])
@pytest.mark.parametrize("pinned", [True, False])
def test_folded_networks(oracle, dm, variant, pinned):
    tables = [workloads.fused_table_u8(ROWS, D, 3, t) for t in range(T)]
    dm.add_network(network("net", tables, variant))
    buf = dm.io_buffer if pinned else (lambda shape, dt: np.zeros(shape, dt))
    io = {"idx": buf((T, CAP), np.int32), "len": buf((T, B), np.int32), "out": buf((B, T * D + 8), np.float32),
          "extra": buf((B, D), np.float32)}
    for request in range(4):              # launch by launch, captured, replayed
        io["idx"][:], io["out"][:], io["extra"][:] = 0, -1, 0
        pooled = []
        for t in range(T):
            l, i, _ = workloads.bags_poisson(B, 6, 0, 12, ROWS, 10 + request, t, np.int32)
            io["len"][t], io["idx"][t, :i.size] = l, i
            w = np.ones(CAP, np.float32)
            if variant == "splat_written":
                w[:CAP // 2] = 0.5
            pooled.append(oracle.frwq_slws_u8_f32(tables[t], w[:i.size], i.astype(np.int64), l))
        dm.run_function("net", io)
        want = np.full((B, T * D + 8), -1, np.float32)
        for t in range(T):
            at = t * D + (0 if variant != "overlapping" else -8 * t)
            want[:, at:at + D] = pooled[t]
        if variant == "twice":
            want[:, T * D - 8:T * D + 8] = pooled[0]
        np.testing.assert_allclose(io["out"], want, rtol=1e-5, atol=1e-5)
        if variant == "read_elsewhere":
            np.testing.assert_allclose(io["extra"], pooled[1], rtol=1e-5, atol=1e-5)
    # a bad request is an error, and the next one is clean
    io["idx"][0, 0] = ROWS
    io["len"][0, 0] = 1
    with pytest.raises(Exception, match="invalid sparse input"):
        dm.run_function("net", io, outputs={"out"})
    io["idx"][0, 0] = 0
    dm.run_function("net", io, outputs={"out"})


def test_bindings_that_change_during_the_call(dm):
    """The request is of the names and arrays that were bound when it was made, whatever becomes of the dict."""
    tables = [workloads.fused_table_u8(ROWS, D, 3, t) for t in range(T)]
    dm.add_network(network("net", tables, "plain"))
    make = lambda: {"".join(["i", "dx"]): np.zeros((T, CAP), np.int32), "".join(["le", "n"]): np.full((T, B), 2, np.int32),
                    "".join(["o", "ut"]): np.full((B, T * D + 8), -1, np.float32)}
    want = make()
    dm.run_function("net", want, outputs={"out"})
    assert (want["out"][:, :T * D] != -1).any()

    class Emptying:
        def __contains__(self, name):
            io.clear()
            return name == "out"

    io = make()
    out = io["out"]
    dm.run_function("net", io, outputs=Emptying())
    assert not io
    np.testing.assert_array_equal(out, want["out"])
