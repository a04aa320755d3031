"""The gather-pool that copies whole rows into shared memory, at its edges: rows at every alignment and the last of a
table, bags round the 32 rows of a step, empty ones, runs cut anywhere, rows that are not there, widths that only it
takes.  Every bag against the bits that the bag gives when it is pooled alone, by another kernel where there is one, and
against float64."""
import numpy as np
import pytest
import torch

from glow_b200 import ops
from test_slws_runs_gpu import DEV, EDGES, check, dev, make_table, pool, want_and_size, with_4bit_surplus

pytestmark = pytest.mark.gpu


def request_of(rng, rows, bags, kind, idt=np.int64):
    lengths = rng.choice(EDGES[:24] + [40, 40, 90], bags).astype(np.int32)
    n = int(lengths.sum())
    idx = rng.integers(0, rows, n).astype(idt)
    idx[rng.integers(0, n, n // 7)] = rows - 1   # the last row ends the table: its last piece is cut
    return lengths, idx, rng.normal(0, 1, n).astype(np.float16 if kind & 1 else np.float32)


def check_pooled(table, kind, dim, w, idx, lengths, got):
    want, size = want_and_size(table, kind, dim, w, idx, lengths)
    check(got.cpu().numpy(), want, with_4bit_surplus(size, table, kind, w, idx, lengths), 2e-3 if kind & 1 else 1e-5)


@pytest.mark.parametrize("kind,dim", [(0, 40), (0, 48), (0, 64), (0, 72), (0, 96), (0, 128), (1, 48), (1, 88), (1, 128),
                                      (2, 40), (2, 56), (2, 96), (2, 128), (2, 136), (2, 256), (3, 48), (3, 104), (3, 192), (3, 256)])
@pytest.mark.parametrize("bags,rows", [(10_000, 1), (20_000, 37), (37_000, 5000)])
def test_single_tables(kind, dim, bags, rows):
    """(above 2048 bags of 57..64 columns another kernel's: those go in tables of 2048 below)"""
    rng = np.random.default_rng(bags + dim + kind)
    table = make_table(kind, rows, dim, 5)
    lengths, idx, w = request_of(rng, rows, bags, kind, np.int32 if kind & 1 else np.int64)
    d = dev(table)
    st = ops.new_status(DEV)
    whole = pool(d, w, idx, lengths, kind, status=st)
    assert int(st.item()) == 0
    ends = np.cumsum(lengths)
    for b in list(range(30)) + list(rng.integers(0, bags, 10)) + [bags - 1]:
        e, l = int(ends[b]), int(lengths[b])
        assert torch.equal(pool(d, w[e - l:e], idx[e - l:e], lengths[b:b + 1], kind)[0], whole[b])
    few = 600
    check_pooled(table, kind, dim, w[:ends[few - 1]], idx[:ends[few - 1]], lengths[:few], whole[:few])


@pytest.mark.parametrize("kind,dim,shift", [(0, 96, 8), (0, 96, 4), (0, 100, 4), (1, 96, 12), (2, 96, 4), (3, 128, 4), (2, 240, 8)])
def test_tables_at_any_four_bytes(kind, dim, shift):
    rng = np.random.default_rng(shift)
    table = make_table(kind, 900, dim, 5)
    lengths, idx, w = request_of(rng, 900, 12_000, kind)
    assert torch.equal(pool(dev(table, shift), w, idx, lengths, kind), pool(dev(table), w, idx, lengths, kind))


@pytest.mark.parametrize("rows", [1, 2, 40])
@pytest.mark.parametrize("kind,dim", [(0, 40), (0, 96), (0, 100), (1, 128), (2, 96), (3, 128)])
@pytest.mark.parametrize("shift", [4, 8, 12])
def test_the_first_row_of_a_table_off_sixteen_bytes(kind, dim, rows, shift):
    """Its first piece begins in front of the table, and what lies there is not read."""
    rng = np.random.default_rng(rows + shift)
    table = make_table(kind, rows, dim, 5)
    lengths, idx, w = request_of(rng, rows, 13_000, kind)
    idx[rng.integers(0, idx.size, idx.size // 5)] = 0
    assert torch.equal(pool(dev(table, shift), w, idx, lengths, kind), pool(dev(table), w, idx, lengths, kind))


@pytest.mark.parametrize("kind,dim,strides", [(0, 40, (128, 192, 208)), (0, 64, (128, 192, 208)), (0, 96, (144, 256, 288, 304)), (1, 96, (256, 288, 304)),
                                              (2, 56, (128, 192, 208)), (2, 96, (192, 288, 304)), (3, 56, (192, 208)), (3, 256, (256, 288, 304))])
def test_rows_stored_apart(kind, dim, strides):
    """Up to so many pieces to a row they are copied whole, padding and all; beyond, another kernel reads their columns."""
    rng = np.random.default_rng(dim)
    table = make_table(kind, 800, dim, 5)
    lengths, idx, w = request_of(rng, 800, 13_000, kind)
    want = pool(dev(table), w, idx, lengths, kind)
    for stride in strides:
        apart = ops.pad_fused_rows(dev(table), kind, stride)
        assert torch.equal(pool(apart, w, idx, lengths, kind, out_line=dim), want)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("dim", [44, 60, 68, 100, 124])
@pytest.mark.parametrize("bags", [1, 7, 300, 2049, 15_000])
def test_widths_off_the_eights(oracle, kind, dim, bags):
    """The operations of the any-shape kernel, which has them otherwise, in the reference's order: bit for bit."""
    rng = np.random.default_rng(bags + dim)
    table = make_table(kind, 700, dim, 9)
    lengths, idx, w = request_of(rng, 700, bags, kind, np.int32)
    lengths[0] = max(1, lengths[0])
    n = int(lengths.sum())
    idx, w = np.resize(idx, n) if idx.size else np.zeros(n, np.int32), np.resize(w, n) if w.size else np.ones(n, w.dtype)
    d = dev(table)
    whole = pool(d, w, idx, lengths, kind)
    few = min(bags, 400)
    e = int(lengths[:few].sum())
    want = oracle.frwq_slws_interp(table, kind, w[:e], idx[:e], lengths[:few])
    np.testing.assert_array_equal(whole[:few].cpu().numpy().view(np.uint8), want.view(np.uint8))
    padded = ops.pad_fused_rows(d, kind, 256)
    assert torch.equal(ops.fused_rowwise_quantized_sparse_lengths_weighted_sum(padded, dev(w), dev(idx), dev(lengths), kind, out_line=dim), whole)


@pytest.mark.parametrize("kind,dim", [(0, 64), (0, 128), (3, 128)])
def test_rows_that_are_not_there(kind, dim):
    """Indices outside the table, a table without rows, negative lengths and lengths beyond the indices."""
    rng = np.random.default_rng(dim)
    rows, bags, tables = 300, 1900, 8
    table = make_table(kind, rows, dim, 5)
    dt = np.float16 if kind & 1 else np.float32
    lengths = rng.integers(0, 40, (tables, bags)).astype(np.int32)
    idx = [rng.integers(0, rows, int(l.sum())) for l in lengths]
    w = [rng.normal(0, 1, i.size).astype(dt) for i in idx]
    bad = [i.copy() for i in idx]
    for i in bad:
        i[::11] = rows + 5
        i[::17] = -3
    d, out = dev(table), torch.empty((tables, bags, dim), dtype=torch.float16 if kind & 1 else torch.float32, device=DEV)
    st = ops.new_status(DEV)

    def run(indices, weights, lens, data=None):
        b = ops.SlwsBatch(kind, table.shape[1], torch.int64, device=DEV)
        b.bind([d if data is None else data] * tables, [dev(x) for x in weights], [dev(x) for x in indices], [dev(x) for x in lens], list(out))
        b.run(st)
        return out.clone()

    with_bad = run(bad, w, lengths)
    assert int(st.item()) == ops.STATUS_INDEX_OUT_OF_RANGE
    st.zero_()
    nothing = [np.where((i >= 0) & (i < rows), x, 0).astype(dt) for i, x in zip(bad, w)]
    there = [np.where((i >= 0) & (i < rows), i, 0) for i in bad]
    clean = run(there, nothing, lengths)
    assert int(st.item()) == 0 and torch.equal(with_bad.float(), clean.float())   # (a zero sum may have either sign)
    none = run(bad, w, lengths, d[:0])
    assert int(st.item()) == ops.STATUS_INDEX_OUT_OF_RANGE and not none.any()
    st.zero_()
    odd = lengths.copy()
    odd[:, 5], odd[:, -1] = -4, odd[:, -1] + 60
    run(idx, w, odd)
    assert int(st.item()) == (ops.STATUS_NEGATIVE_LENGTH | ops.STATUS_LENGTHS_OVERRUN)


@pytest.mark.parametrize("kind,dim", [(0, 40), (0, 72), (0, 88), (0, 128), (2, 128), (2, 256), (3, 104)])
@pytest.mark.parametrize("rows_of_a_bag", [33, 64, 65])
def test_the_first_steps_of_a_run(kind, dim, rows_of_a_bag):
    """The second step of a run is asked for right behind the first, by lanes that do not leave the first's copies together
    (3 to 9 pieces to a row, so that 0 to 5 lanes copy none): each step of 32 rows has a number range of its own, and a row
    fetched by the other step's number is not in the sums."""
    rng = np.random.default_rng(dim + rows_of_a_bag)
    rows, bags = 4096, 30_000
    table = make_table(kind, rows, dim, 5)
    lengths = np.full(bags, rows_of_a_bag, np.int32)
    step = np.arange(rows_of_a_bag) // 32
    idx = (rng.integers(0, rows // 4, (bags, rows_of_a_bag)) + step * (rows // 4)).reshape(-1)
    w = rng.normal(0, 1, idx.size).astype(np.float16 if kind & 1 else np.float32)
    got = pool(dev(table), w, idx, lengths, kind)
    few = 300
    check_pooled(table, kind, dim, w[:few * rows_of_a_bag], idx[:few * rows_of_a_bag], lengths[:few], got[:few])
    for b in (0, 1, 17, bags - 1):
        at = slice(b * rows_of_a_bag, (b + 1) * rows_of_a_bag)
        assert torch.equal(pool(dev(table), w[at], idx[at], lengths[:1], kind)[0], got[b])


@pytest.mark.parametrize("kind,dim", [(0, 96), (1, 96), (2, 96), (3, 128), (0, 100)])
def test_weights_of_rows_that_are_not_there(kind, dim):
    """A row that is not there adds nothing, whatever its weight: a NaN or an infinity of an index outside the table (or of
    another shard's row) is in no sum, nor is what a lane beyond the end of a bag had in its register."""
    rng = np.random.default_rng(dim + kind)
    rows, bags = 500, 13_000
    table = make_table(kind, rows, dim, 5)
    d = dev(table)
    dt = np.float16 if kind & 1 else np.float32
    lengths = rng.integers(0, 75, bags).astype(np.int32)
    n = int(lengths.sum())
    idx, w = rng.integers(0, rows, n), rng.normal(0, 1, n).astype(dt)
    out = rng.random(n) < 0.2
    bad_i, bad_w, there, nothing = idx.copy(), w.copy(), idx.copy(), w.copy()
    bad_i[out] = rng.choice([rows, rows + 9, -1], out.sum())
    bad_w[out] = rng.choice(np.array([np.nan, np.inf, -np.inf, 1.0], dt), out.sum())
    there[out], nothing[out] = 0, 0
    st = ops.new_status(DEV)
    got = pool(d, bad_w, bad_i, lengths, kind, status=st)
    assert int(st.item()) == ops.STATUS_INDEX_OUT_OF_RANGE
    want = pool(d, nothing, there, lengths, kind)
    assert bool(torch.isfinite(want).all()) and torch.equal(got.float(), want.float())   # (a zero sum may have either sign)
    few = 500   # and the kernel of small launches
    few_n = int(lengths[:few].sum())
    assert torch.equal(pool(d, bad_w[:few_n], bad_i[:few_n], lengths[:few], kind).float(), want[:few].float())
    # offsets that go backwards: every bag is a stream of its own, and the rows behind its end have weights of before
    mean = 37
    begins = np.arange(bags + 1, dtype=np.int64) % 200 * mean
    begins[1::2] += 40   # bags of 77 rows, and ones that end before they begin
    weights = w[:begins.max() + 1].copy()
    weights[rng.random(weights.size) < 0.002] = np.nan
    out = ops.embedding_bag_byte_rowwise_offsets(d, dev(weights), dev(idx[:weights.size]), dev(begins), kind, has_end_offset=True, status=st)
    for b in range(0, 400):
        at, to = int(begins[b]), max(int(begins[b]), int(begins[b + 1]))
        alone = pool(d, weights[at:to], idx[at:to], np.int32([to - at]), kind)[0]
        assert torch.equal(torch.nan_to_num(out[b].float(), nan=1e30), torch.nan_to_num(alone.float(), nan=1e30)), b


@pytest.mark.parametrize("kind,dim", [(0, 96), (2, 128)])
def test_weights_of_other_shards_rows(kind, dim):
    rng = np.random.default_rng(dim)
    rows, bags, tables, shards = 300, 1900, 8, 4
    table = make_table(kind, rows, dim, 5)
    d = dev(table)
    lengths = rng.integers(0, 60, (tables, bags)).astype(np.int32)
    idx = [rng.integers(0, rows * shards, int(l.sum())) for l in lengths]
    mine = [(i >= rows) & (i < 2 * rows) for i in idx]
    w = [np.where(m, rng.normal(0, 1, m.size), np.inf).astype(np.float32) for m in mine]
    out = torch.empty((tables, bags, dim), device=DEV)
    st = ops.new_status(DEV)
    b = ops.SlwsBatch(kind, table.shape[1], torch.int64, device=DEV)
    b.bind([d] * tables, [dev(x) for x in w], [dev(x) for x in idx], [dev(x) for x in lengths], list(out), row_ranges=[(rows, rows * shards)] * tables)
    b.run(st)
    assert int(st.item()) == 0
    for i in range(tables):
        want = pool(d, np.where(mine[i], w[i], 0).astype(np.float32), np.where(mine[i], idx[i] - rows, 0), lengths[i], kind)
        assert torch.equal(out[i], want)
