"""The gather-pool's runs of bags at their edges: bags of every length round the 4, 8 and 16 rows of a
step, among short and empty ones; every width and row alignment the kernel is built for; launches on
both sides of the sizes where it changes its step, its runs and where bag boundaries come from; weights
of very different sizes; rows that are not finite.  Against a float64 restatement of the operator."""
import numpy as np
import pytest
import torch

from glow_b200 import ops, workloads

pytestmark = pytest.mark.gpu
DEV = "cuda"
EDGES = [0, 1, 2, 31, 32, 33, 5, 0, 0, 7, 9, 3, 1, 1, 63, 64, 65, 255, 256, 257, 0, 288, 600, 15, 16, 17, 30, 2, 1, 4, 8, 0]


def make_table(kind, rows, dim, seed):
    f = workloads.fused_table_u4 if kind >= 2 else workloads.fused_table_u8
    return f(rows, dim, seed, 0, fp16_scale_offset=bool(kind & 1))


def want_and_size(table, kind, dim, w, idx, lengths):
    tail = 4 if kind & 1 else 8
    so = table[:, -tail:].copy().view(np.float16 if kind & 1 else np.float32).astype(np.float64)
    q = table[:, :dim if kind < 2 else dim // 2]
    if kind >= 2:
        q = np.stack([q & 15, q >> 4], 2).reshape(len(table), dim)
    q, sc, of = q.astype(np.float64), so[:, :1], so[:, 1:]
    w = np.asarray(w, np.float64)[:, None]
    # (the kernel's association: where a weight is infinite, w * scale * q and w * offset may cancel)
    terms, size = (w * sc[idx]) * q[idx] + w * of[idx], np.abs(w) * (np.abs(sc[idx] * q[idx]) + np.abs(of[idx]))
    ends = np.cumsum(lengths)
    return (np.stack([terms[e - l:e].sum(0) for l, e in zip(lengths, ends)]),
            np.stack([size[e - l:e].sum(0) for l, e in zip(lengths, ends)]))


def dev(a, shift=0):
    """The array on the device, `shift` bytes behind a 16-byte boundary."""
    a = np.ascontiguousarray(a)
    buf = torch.zeros(a.nbytes + 32, dtype=torch.uint8, device=DEV)
    at = -buf.data_ptr() % 16 + shift
    view = buf[at:at + a.nbytes].view(torch.from_numpy(a).dtype).view(a.shape)
    view.copy_(torch.from_numpy(a))
    return view


def check(got, want, size, rel):
    bound = rel * np.maximum(size, np.abs(want)) + 1e-30
    err = np.abs(got.astype(np.float64) - want)
    assert (err <= bound).all(), "largest error / bound %g" % np.max(err / bound)


def pool(table, w, idx, lengths, kind, **kw):
    return ops.fused_rowwise_quantized_sparse_lengths_weighted_sum(table, dev(w), dev(idx), dev(lengths), kind, **kw)


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("dim", [8, 16, 24, 32, 40, 64, 96, 128, 136, 256, 1000])
def test_lengths_widths_and_alignments(kind, dim):
    rng = np.random.default_rng(dim + kind)
    rows = 700
    table = make_table(kind, rows, dim, dim)
    lengths = np.concatenate([EDGES, rng.integers(0, 9, 40), rng.permutation(EDGES)]).astype(np.int32)
    n = int(lengths.sum())
    idx = rng.integers(0, rows, n)
    w = rng.normal(0, 1, n).astype(np.float16 if kind & 1 else np.float32)
    want, size = want_and_size(table, kind, dim, w, idx, lengths)
    status = ops.new_status(DEV)
    first = None
    for shift in (0, 4, 1, 2, 8):
        for idt in (np.int64, np.int32):
            got = pool(dev(table, shift), w, idx.astype(idt), lengths, kind, status=status)
            first = got if first is None else first
            assert torch.equal(got, first)   # neither the alignment nor the index type shows
    check(first.cpu().numpy(), want, size, 2e-3 if kind & 1 else 1e-5)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    got = ops.embedding_bag_byte_rowwise_offsets(dev(table), dev(w), dev(idx.astype(np.int64)), dev(offsets), kind, status=status)
    assert torch.equal(got, first)
    assert int(status.item()) == 0


@pytest.mark.parametrize("bags", [1, 3, 2048, 2049, 9000, 120_000])
@pytest.mark.parametrize("kind,dim", [(0, 64), (3, 128)])
def test_launch_size_does_not_show(bags, kind, dim):
    """A bag pooled beside any number of others gives the same bits as pooled alone."""
    rng = np.random.default_rng(bags)
    table = dev(make_table(kind, 5000, dim, 3))
    lengths = rng.choice(EDGES if bags < 10_000 else [0, 1, 2, 5, 9, 33], bags).astype(np.int32)
    lengths[-1] = 300
    n = int(lengths.sum())
    idx, w = rng.integers(0, 5000, n), rng.normal(0, 1, n).astype(np.float16 if kind & 1 else np.float32)
    whole = pool(table, w, idx, lengths, kind)
    ends = np.cumsum(lengths)
    for b in [0, bags - 1] + list(rng.integers(0, bags, 12)):
        e, l = int(ends[b]), int(lengths[b])
        assert torch.equal(pool(table, w[e - l:e], idx[e - l:e], lengths[b:b + 1], kind)[0], whole[b])


@pytest.mark.parametrize("kind", [0, 2])
def test_weights_of_changing_size(kind):
    rng = np.random.default_rng(5)
    table = make_table(kind, 300, 64, 9)
    lengths = np.array([200, 33, 500, 64, 32, 8], np.int32)
    n = int(lengths.sum())
    idx = rng.integers(0, 300, n)
    w = rng.normal(0, 1, n) * 10.0 ** rng.integers(-8, 8, n)
    w[200:233] = 0
    w[232] = 1.5
    w[233:300] = 1e-30
    w = w.astype(np.float32)
    want, size = want_and_size(table, kind, 64, w, idx, lengths)
    check(pool(dev(table), w, idx, lengths, kind).cpu().numpy(), want, size, 1e-5)


@pytest.mark.parametrize("dim", [64, 136])
def test_rows_that_are_not_finite(dim):
    """Infinite and undefined scales, offsets and weights reach exactly the bags they belong to."""
    rng = np.random.default_rng(7)
    table = make_table(0, 400, dim, 11)
    sc = table[:, -8:].copy().view(np.float32)
    sc[3, 0], sc[4, 1], sc[5, 0], sc[6, 1] = np.inf, -np.inf, np.nan, np.nan
    table[:, -8:] = sc.view(np.uint8)
    lengths = np.array([5, 3, 40, 2, 100, 1, 7, 33, 6, 300], np.int32)
    n = int(lengths.sum())
    idx = rng.integers(10, 400, n)
    w = rng.normal(0, 1, n).astype(np.float32)
    ends = np.cumsum(lengths)
    for b, r in ((1, 3), (2, 4), (4, 5), (7, 6), (9, 3)):
        idx[ends[b] - 1] = r
    w[ends[3] - 1] = np.inf
    table[3, :8] = 0                        # an infinite scale times a zero byte is undefined
    with np.errstate(all="ignore"):
        want, size = want_and_size(table, 0, dim, w, idx, lengths)
    got = pool(dev(table), w, idx, lengths, 0).cpu().numpy()
    fine = np.isfinite(want)
    assert (np.isnan(got) == np.isnan(want)).all() and (got[np.isinf(want)] == want[np.isinf(want)]).all()
    assert fine.any(1).sum() == 4
    check(got[fine], want[fine], size[fine], 1e-5)


@pytest.mark.parametrize("kind,dim", [(0, 64), (2, 64), (2, 40), (1, 192), (3, 256)])
@pytest.mark.parametrize("bags", [600, 5000, 20_000, 70_000])
def test_launches_of_every_tier_agree(bags, kind, dim):
    """Sixteen, eight and four rows per step, one chunk per lane and several, runs of one bag per group and of more:
    the same bits as the bag pooled alone."""
    rng = np.random.default_rng(bags + dim)
    table = dev(make_table(kind, 3000, dim, 3))
    lengths = rng.choice([0, 1, 3, 7, 8, 9, 16, 17, 40], bags).astype(np.int32)
    lengths[bags // 2] = 200
    n = int(lengths.sum())
    idx, w = rng.integers(0, 3000, n), rng.normal(0, 1, n).astype(np.float16 if kind & 1 else np.float32)
    whole = pool(table, w, idx, lengths, kind)
    ends = np.cumsum(lengths)
    for b in [0, bags // 2, bags - 1] + list(rng.integers(0, bags, 5)):
        e, l = int(ends[b]), int(lengths[b])
        assert torch.equal(pool(table, w[e - l:e], idx[e - l:e], lengths[b:b + 1], kind)[0], whole[b])


def with_4bit_surplus(size, table, kind, w, idx, lengths):
    """`size`, such that 1e-5 of it also holds what a bag of 4-bit rows may be off by that has q = 0 and hardly an
    offset: the columns are summed as 128 * w * scale * (1 + q / 128) and the ones taken out again, two roundings of
    2^-24 of sums of that size."""
    if kind < 2:
        return size
    so = table[:, -(4 if kind & 1 else 8):].copy().view(np.float16 if kind & 1 else np.float32).astype(np.float64)
    terms = np.concatenate([[0], np.cumsum(128 * np.abs(np.asarray(w, np.float64) * so[idx, 0])[:int(np.sum(lengths))])])
    ends = np.cumsum(lengths)
    return size + 1e5 * 2.0 ** -23 * (terms[ends] - terms[ends - lengths])[:, None]


@pytest.mark.parametrize("kind,dim", [(0, 48), (1, 64), (2, 40), (3, 64), (2, 96), (3, 128), (2, 136), (3, 256), (1, 128)])
@pytest.mark.parametrize("bags", [700, 2500, 6000])
def test_tables_of_every_skew_in_one_launch(kind, dim, bags):
    """Even tables, skewed ones, an empty one and one of a single long bag, pooled by one launch whose tables may take
    different kernels: the sums of the operator, and the bits of each table pooled alone."""
    rng = np.random.default_rng(dim + bags)
    laws = [rng.integers(18, 23, bags), rng.choice(EDGES[:24] + [200] * 2, bags), np.zeros(bags, int),
            np.eye(1, bags, bags // 3, dtype=int)[0] * 600, rng.integers(0, 3, bags)]
    tables, w, idx, lengths, alone = [], [], [], [], []
    status = ops.new_status(DEV)
    for law in laws:
        t, l = make_table(kind, 900, dim, len(tables)), law.astype(np.int32)
        n = int(l.sum())
        i, x = rng.integers(0, 900, n + 1), rng.normal(0, 1, n + 1).astype(np.float16 if kind & 1 else np.float32)
        tables.append(dev(t)), w.append(dev(x)), idx.append(dev(i)), lengths.append(dev(l))
        alone.append(pool(tables[-1], x, i, l, kind, status=status))
        want, size = want_and_size(t, kind, dim, x, i, l)
        size = with_4bit_surplus(size, t, kind, x, i, l)
        check(alone[-1].cpu().numpy(), want, size, 2e-3 if kind & 1 else 1e-5)
    out = torch.full((len(laws), bags, dim), 7.0, dtype=alone[0].dtype, device=DEV)
    batch = ops.SlwsBatch(kind, tables[0].shape[1], torch.int64, device=DEV)
    batch.bind(tables, w, idx, lengths, list(out)).run(status)
    for programmatic in (False, True):
        with ops.programmatic_launch(programmatic):
            batch.run(status)
        for got, one in zip(out, alone):
            assert torch.equal(got, one)
        out.fill_(7.0)
    assert int(status.item()) == 0


@pytest.mark.parametrize("kind,dim", [(0, 64), (3, 96), (2, 256)])
@pytest.mark.parametrize("bags", [60, 4000, 15_000])
def test_offsets_that_go_backwards_and_rows_that_are_not_there(kind, dim, bags):
    """Bags with a start above their end are empty and reported; others are pooled from where they begin."""
    rng = np.random.default_rng(bags)
    table = make_table(kind, 500, dim, 2)
    lengths = rng.choice([0, 1, 5, 17, 33, 64, 130], bags)
    offsets = np.concatenate([[0], np.cumsum(lengths)])
    n = int(offsets[-1])
    for b in rng.integers(1, bags, 8):
        offsets[b] = rng.integers(0, n)
    idx = rng.integers(0, 500, n)
    idx[::97], idx[::89] = 500, -1
    w = rng.normal(0, 1, n).astype(np.float16 if kind & 1 else np.float32)
    w64, good = np.where((idx >= 0) & (idx < 500), w, 0), np.clip(idx, 0, 499)
    spans = [np.arange(a, b) for a, b in zip(offsets[:-1], offsets[1:])]
    rows, sizes = np.concatenate(spans), np.array([len(s) for s in spans])
    want, size = want_and_size(table, kind, dim, w64[rows], good[rows], sizes)
    size = with_4bit_surplus(size, table, kind, w64[rows], good[rows], sizes)
    status = ops.new_status(DEV)
    got = ops.embedding_bag_byte_rowwise_offsets(dev(table), dev(w), dev(idx), dev(offsets), kind, status=status)
    check(got.cpu().numpy(), want, size, 2e-3 if kind & 1 else 1e-5)
    assert int(status.item()) & (ops.STATUS_BAD_OFFSETS | ops.STATUS_INDEX_OUT_OF_RANGE) == int(status.item()) != 0


@pytest.mark.parametrize("bags", [2049, 3000, 40_000])
@pytest.mark.parametrize("skewed", [False, True])
def test_both_forms_know_a_skewed_table(bags, skewed):
    """The word behind the boundaries of a table, by which its kernel is chosen, from lengths and from offsets."""
    rng = np.random.default_rng(bags)
    lengths = rng.integers(10, 14, bags).astype(np.int32)
    if skewed:
        lengths[rng.choice(bags, bags // 50, replace=False)] = 150
    n = int(lengths.sum())
    table, idx, w = make_table(0, 400, 64, 1), rng.integers(0, 400, n), rng.normal(0, 1, n).astype(np.float32)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    got = []
    for form, bounds in ((ops.fused_rowwise_quantized_sparse_lengths_weighted_sum, lengths), (ops.embedding_bag_byte_rowwise_offsets, offsets)):
        ws = torch.full((ops.slws_workspace_bytes(bags),), 255, dtype=torch.uint8, device=DEV)
        got.append(form(dev(table), dev(w), dev(idx), dev(bounds), 0, workspace=ws))
        words = ws.view(torch.int64)[:bags + 2].cpu().numpy()
        np.testing.assert_array_equal(words[:-1], offsets)
        assert words[-1] == (150 if skewed else 0)
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("kind,dim", [(0, 16), (3, 64)])
def test_index_arrays_too_long_to_count(kind, dim):
    """An index array of more entries than the kernels count takes the kernel that counts in 64 bits.  (The bags are
    short and lie at its beginning: only its length, which bounds them and nothing else, is that large.)"""
    import ctypes as C

    from glow_b200 import _lib
    rng = np.random.default_rng(1)
    table, lengths = make_table(kind, 300, dim, 4), rng.integers(0, 40, 33).astype(np.int32)
    n, dt = int(lengths.sum()), torch.float16 if kind & 1 else torch.float32
    idx, w = rng.integers(0, 300, n), rng.normal(0, 1, n).astype(np.float16 if kind & 1 else np.float32)
    want, size = want_and_size(table, kind, dim, w, idx, lengths)
    size = with_4bit_surplus(size, table, kind, w, idx, lengths)
    held, status = (dev(table), dev(w), dev(idx), dev(lengths)), ops.new_status(DEV)
    ws = torch.empty(ops.slws_workspace_bytes(33), dtype=torch.uint8, device=DEV)
    p = lambda a: C.c_void_p(a.data_ptr())
    for claimed in (n, 2 ** 31 // 7 * 4 + 8, 2 ** 31 + 1):
        out = torch.empty((33, dim), dtype=dt, device=DEV)
        _lib.check(_lib.lib().glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum(
            p(out), p(held[0]), kind, 300, p(held[1]), p(held[2]), 1, p(held[3]), 33, claimed, table.shape[1], dim,
            int(dt == torch.float16), 0, p(ws), ws.numel(), p(status), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        check(out.cpu().numpy(), want, size, 2e-3 if kind & 1 else 1e-5)
    assert int(status.item()) == 0


@pytest.mark.parametrize("kind,dim", [(0, 64), (0, 96), (2, 128), (0, 192), (3, 256)])
@pytest.mark.parametrize("tables,bags,mean", [(3, 591, 7), (3, 592, 9), (3, 593, 9), (5, 400, 20), (4, 700, 3), (2, 2100, 12), (3, 2100, 30)])
def test_kernels_chosen_by_the_rows_of_a_launch_agree(kind, dim, tables, bags, mean):
    """Bags of a few rows and of more, on both sides of the launch sizes at which the length of bags decides: a caller who
    says how many rows there are, one who does not, and one table at a time get the same bits."""
    g = np.random.Generator(np.random.PCG64(tables * bags + mean))
    dt = ops.result_dtype(kind)
    data = [dev(make_table(kind, 500, dim, 20 + t)) for t in range(tables)]
    lengths = [g.poisson(mean, bags).astype(np.int32) for _ in range(tables)]
    lengths[0][1::9] = 0
    lengths[1][5] = 150
    idx = [dev(g.integers(0, 500, int(l.sum()))) for l in lengths]
    w = [torch.rand(len(i), device=DEV).to(dt) for i in idx]
    ln = [dev(l) for l in lengths]
    out = torch.zeros((tables, bags, dim), dtype=dt, device=DEV)
    status = ops.new_status(DEV)
    batch = ops.SlwsBatch(kind, data[0].shape[1], torch.int64, device=DEV)
    batch.bind(data, w, idx, ln, list(out))
    batch.run(status)
    known = out.clone()
    out.zero_()
    batch.num_indices = -1
    batch.run(status)
    one = torch.stack([ops.fused_rowwise_quantized_sparse_lengths_weighted_sum(*a, kind) for a in zip(data, w, idx, ln)])
    assert torch.equal(out, known) and torch.equal(one, known) and int(status.item()) == 0
