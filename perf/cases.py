"""The performance cases of the library: the calls its users make, at the sizes they make them.

`listed()` names the cases; `draw(rng)` gives further ones of the same ranges; `prepare(case, seed)`
builds what a program holds before the call (inputs, tables, weights, workspaces, a loaded network);
`run(state)` is one call; `work(case)` what the call cannot do without; `tolerance(case)` how far the
results of another correct implementation may be off.

Every case has a "path":
  pool      one embedding gather-pool node (lengths or offsets form) over one fused-rowwise table
  tables    many tables of one row width pooled by one launch (ops.SlwsBatch)
  tbe       table-batched embedding bags over one byte buffer (IntNBitSplitEmbeddingBags)
  fc        int8 fully connected layers and matrix products, static and dynamic quantization
  resnet    the int8 ResNet-50, fp32 NCHW images to logits
  dlrm      one step of the recommendation model on one GPU
  request   the recommendation model as a network in the device manager, host buffers in and out
"""
import functools
import math

import numpy as np
import torch

from glow_b200 import dlrm, ops, resnet, runtime

DEV = "cuda"
KINDS = {"u8": ops.UINT8_FUSED, "u8_fp16": ops.UINT8_FUSED_FP16, "u4": ops.UINT4_FUSED, "u4_fp16": ops.UINT4_FUSED_FP16}
TBE_TYPES = {"fp32": ops.EST_FLOAT, "fp16": ops.EST_FLOAT16, "int8": ops.EST_INT8, "int4": ops.EST_INT4}


def listed():
    return [
        # One SparseLengthsWeightedSum node of an inference graph, run on its own with ops' defaults: the first
        # benchmark configuration (1,000,000 x 64 uint8, 1024 bags of Poisson(32)).  The smallest pooling call.
        {"name": "pool_one_node", "path": "pool", "kind": "u8", "rows": 1_000_000, "dim": 64, "bags": 1024, "mean": 32,
         "idx64": True, "form": "lengths"},
        # The benchmark's headline launch: 256 such tables at once.  The largest pooling call.
        {"name": "pool_256_tables", "path": "tables", "kind": "u8", "tables": 256, "rows": 1_000_000, "dim": 64,
         "bags": 1024, "mean": 32, "law": "poisson", "idx64": True},
        # The 4-bit sweep's middle width: 10,000,000-row tables, fp16 scales, weights and result, 8192 bags.
        {"name": "pool_4bit_tables", "path": "tables", "kind": "u4_fp16", "tables": 4, "rows": 10_000_000, "dim": 128,
         "bags": 8192, "mean": 64, "law": "poisson", "idx64": True},
        # Table-batched bags as the benchmark's default: int4 rows of 128 columns, Poisson(64), fp16 result.
        {"name": "table_batched_bags", "path": "tbe", "type": "int4", "tables": 8, "rows": 2_000_000, "dim": 128,
         "bags": 8192, "mean": 64, "idx64": True, "weighted": False, "mean_pooling": False, "out_fp16": True},
        # A hidden layer of a model that answers a few requests at a time: latency of one small launch.
        {"name": "fc_small", "path": "fc", "form": "rowwise", "m": 8, "k": 1024, "n": 1024, "asym": False, "relu": True},
        # The second benchmark configuration: the large int8 layer.
        {"name": "fc_large", "path": "fc", "form": "rowwise", "m": 2048, "k": 4096, "n": 4096, "asym": False,
         "relu": False},
        # The first top layer behind the pairwise dots of 26 tables of 128 columns (128 + 27 * 26 / 2 = 479 inputs),
        # weights quantized with the default, asymmetric, schema: an odd reduction length.
        {"name": "fc_ragged", "path": "fc", "form": "rowwise", "m": 2048, "k": 479, "n": 1024, "asym": True, "relu": True},
        # Dynamically quantized layer (fp16 in and out) at an ordinary batch.
        {"name": "fc_dynamic", "path": "fc", "form": "dynamic", "m": 512, "k": 4096, "n": 4096, "asym": False,
         "relu": False},
        # The third configuration, as a throughput server runs it: batch 64, the network replayed from a CUDA graph.
        {"name": "resnet50_batch64", "path": "resnet", "batch": 64, "size": 224, "graph": True},
        # One image through the same network by its forward call: the latency of one classification.
        {"name": "resnet50_one_image", "path": "resnet", "batch": 1, "size": 224, "graph": False},
        # The fourth configuration's step (64 tables of 128 columns, batch 4096, power-law lengths and rows) with
        # 1,000,000-row tables, so that several models fit one GPU.
        {"name": "dlrm_step", "path": "dlrm", "tables": 64, "rows": 1_000_000, "dim": 128, "batch": 4096, "mean": 40,
         "graph": True},
        # A recommendation request through the device manager's request call: 26 tables, 128 candidates, pinned
        # host buffers in, scores in a host buffer out.
        {"name": "request_recsys", "path": "request", "tables": 26, "rows": 100_000, "dim": 64, "batch": 128, "mean": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["pool", "tables", "tbe", "fc", "fc", "resnet", "dlrm", "request"])
    dims = [16, 32, 48, 64, 96, 100, 128, 192, 256]   # 100 columns: a row that no 16-byte line divides
    if path == "pool":
        c = {"kind": rng.choice(list(KINDS)), "rows": _log(rng, 10_000, 2_000_000), "dim": rng.choice(dims),
             "bags": _log(rng, 16, 4096), "mean": _log(rng, 1, 100), "idx64": rng.random() < 0.5,
             "form": rng.choice(["lengths", "lengths", "offsets"])}
    elif path == "tables":
        c = {"kind": rng.choice(list(KINDS)), "tables": _log(rng, 2, 128), "rows": _log(rng, 50_000, 4_000_000),
             "dim": rng.choice(dims), "bags": _log(rng, 64, 8192), "mean": _log(rng, 1, 64),
             "law": rng.choice(["poisson", "power"]), "idx64": rng.random() < 0.5}
        while c["tables"] * c["rows"] * c["dim"] > 16e9 or c["tables"] * c["bags"] * c["mean"] * c["dim"] > 530e6:
            c["tables"], c["bags"] = max(2, c["tables"] * 2 // 3), max(64, c["bags"] * 3 // 4)
            c["rows"] = max(50_000, c["rows"] * 3 // 4)
    elif path == "tbe":
        c = {"type": rng.choice(list(TBE_TYPES) + ["mixed"]), "tables": _log(rng, 1, 64), "rows": _log(rng, 10_000, 2_000_000),
             "dim": rng.choice([16, 32, 64, 96, 128, 256]), "bags": _log(rng, 16, 8192), "mean": _log(rng, 1, 64),
             "idx64": rng.random() < 0.5, "weighted": rng.random() < 0.5, "mean_pooling": rng.random() < 0.25,
             "out_fp16": rng.random() < 0.5}
        while c["tables"] * c["rows"] * c["dim"] > 2.1e9 or c["tables"] * c["bags"] * c["mean"] * c["dim"] > 530e6:
            c["tables"], c["bags"] = max(1, c["tables"] * 2 // 3), max(16, c["bags"] * 3 // 4)
            c["rows"] = max(10_000, c["rows"] * 3 // 4)
    elif path == "fc":
        form = rng.choice(["rowwise", "rowwise", "tensor", "matmul", "dynamic"])
        c = {"form": form, "m": _log(rng, 1, 2048), "k": _log(rng, 16, 4096), "n": _log(rng, 8, 4096),
             "asym": rng.random() < 0.5, "relu": form == "rowwise" and rng.random() < 0.5}
    elif path == "resnet":
        size = rng.randrange(128, 289)
        c = {"batch": _log(rng, 1, 64), "size": size, "graph": rng.random() < 0.5}
        c["batch"] = max(1, min(c["batch"], 64 * 224 * 224 // (size * size)))
    elif path == "dlrm":
        c = {"tables": _log(rng, 4, 64), "rows": _log(rng, 50_000, 1_000_000), "dim": rng.choice([32, 64, 128]),
             "batch": _log(rng, 16, 4096), "mean": _log(rng, 2, 40), "graph": rng.random() < 0.5}
    else:
        c = {"tables": _log(rng, 4, 40), "rows": _log(rng, 10_000, 200_000), "dim": rng.choice([16, 32, 64, 128]),
             "batch": _log(rng, 1, 1024), "mean": _log(rng, 1, 30)}
    return dict(c, path=path)


# ------------------------------------------------------------------------------------------
# inputs (made on the GPU from the seed)
# ------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * seed + 17)


def _bytes(n, g):
    """n random bytes."""
    words = torch.empty((n + 7) // 4, dtype=torch.int32, device=DEV)
    words.random_(-2 ** 31, 2 ** 31, generator=g)
    return words.view(torch.uint8)[:n]


def _fused_table(rows, dim, kind, g):
    """Random payload, scale U(0.001, 0.01), offset U(-1, 1) per row."""
    line = ops.fused_row_bytes(dim, kind)
    t = _bytes(rows * line, g).view(rows, line)
    so = torch.empty((rows, 2), device=DEV)
    so[:, 0].uniform_(0.001, 0.01, generator=g)
    so[:, 1].uniform_(-1, 1, generator=g)
    so = so.to(torch.float16 if kind & 1 else torch.float32)
    tail = so.view(torch.uint8)
    t[:, line - tail.shape[1]:] = tail
    return t


def _bag_lengths(n, mean, law, g):
    """Poisson(mean) lengths of at least one, or power-law ones on [1, 200] scaled to the mean."""
    if law == "poisson":
        return torch.poisson(torch.full((n,), float(mean), device=DEV), generator=g).clamp_(1, 4 * mean).to(torch.int32)
    ks = np.arange(1, 201, dtype=np.float64)
    raw_mean = float((ks ** -0.05).sum() / (ks ** -1.05).sum())
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    raw = (1 + u * (201.0 ** -0.05 - 1)) ** (1 / -0.05)
    return torch.round(raw * (mean / raw_mean)).clamp_(0, 200).to(torch.int32)


def _rows(n, rows, law, idx64, g):
    """Uniform row numbers, or power-law ones spread over the table by a fixed permutation."""
    if law == "poisson":
        return torch.randint(0, rows, (n,), device=DEV, generator=g, dtype=torch.int64 if idx64 else torch.int32)
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    rank = ((1 + u * ((rows + 1.0) ** -0.05 - 1)) ** (1 / -0.05) - 1).to(torch.int64).clamp_(0, rows - 1)
    mult = 2654435761
    while math.gcd(mult, rows) != 1:
        mult += 2
    return ((rank * mult) % rows).to(torch.int64 if idx64 else torch.int32)


# ------------------------------------------------------------------------------------------
# what a program holds, per path; each returns the call
# ------------------------------------------------------------------------------------------
def _prepare_pool(c, g):
    kind = KINDS[c["kind"]]
    table = _fused_table(c["rows"], c["dim"], kind, g)
    lengths = _bag_lengths(c["bags"], c["mean"], "poisson", g)
    n = int(lengths.sum())
    indices = _rows(n, c["rows"], "poisson", c["idx64"], g)
    weights = torch.rand(n, device=DEV, generator=g).to(ops.result_dtype(kind))
    if c["form"] == "lengths":
        return lambda: ops.fused_rowwise_quantized_sparse_lengths_weighted_sum(table, weights, indices, lengths, kind)
    offsets = torch.zeros(c["bags"] + 1, dtype=indices.dtype, device=DEV)
    offsets[1:] = torch.cumsum(lengths, 0)
    return lambda: ops.embedding_bag_byte_rowwise_offsets(table, weights, indices, offsets, kind)


def _prepare_tables(c, g):
    kind, line = KINDS[c["kind"]], ops.fused_row_bytes(c["dim"], KINDS[c["kind"]])
    dt = ops.result_dtype(kind)
    tables, weights, indices, lengths = [], [], [], []
    for _ in range(c["tables"]):
        tables.append(_fused_table(c["rows"], c["dim"], kind, g))
        lengths.append(_bag_lengths(c["bags"], c["mean"], c["law"], g))
        n = int(lengths[-1].sum())
        indices.append(_rows(n, c["rows"], c["law"], c["idx64"], g))
        weights.append(torch.rand(n, device=DEV, generator=g).to(dt))
    out = torch.empty((c["tables"], c["bags"], c["dim"]), dtype=dt, device=DEV)
    batch = ops.SlwsBatch(kind, line, torch.int64 if c["idx64"] else torch.int32, device=DEV)
    batch.bind(tables, weights, indices, lengths, list(out))
    status = ops.new_status(DEV)

    def call():
        batch.run(status)
        return out

    return call


def _tbe_types(c):
    names = ["fp16", "int8", "int4"] if c["type"] == "mixed" else [c["type"]]
    return [names[t % len(names)] for t in range(c["tables"])]


def _prepare_tbe(c, g):
    T, rows, D, B = c["tables"], c["rows"], c["dim"], c["bags"]
    parts, offs, at = [], [], 0
    for name in _tbe_types(c):
        ty = TBE_TYPES[name]
        line = ops.split_embedding_row_bytes(D, ty)
        if name in ("fp32", "fp16"):
            t = torch.empty((rows, D), dtype=torch.float32 if name == "fp32" else torch.float16, device=DEV)
            t.normal_(0, 1, generator=g)
            flat = torch.zeros((rows, line), dtype=torch.uint8, device=DEV)
            flat[:, :D * t.element_size()] = t.view(torch.uint8)
        else:
            flat = _bytes(rows * line, g).view(rows, line)
            so = torch.empty((rows, 2), device=DEV)
            so[:, 0].uniform_(0.001, 0.01, generator=g)
            so[:, 1].uniform_(-1, 1, generator=g)
            flat[:, :4] = so.to(torch.float16).view(torch.uint8)
        parts.append(flat.view(-1))
        offs.append(at)
        at += flat.numel()
    data = torch.cat(parts)
    del parts
    idt = torch.int64 if c["idx64"] else torch.int32
    lengths = torch.poisson(torch.full((T * B,), float(c["mean"]), device=DEV), generator=g).to(torch.int64)
    offsets = torch.zeros(T * B + 1, dtype=idt, device=DEV)
    offsets[1:] = torch.cumsum(lengths, 0)
    n = int(lengths.sum())
    indices = torch.randint(0, rows, (n,), device=DEV, generator=g, dtype=idt)
    iw = torch.rand(n, device=DEV, generator=g) if c["weighted"] else None
    placements = torch.full((T,), ops.PLACEMENT_HOST, dtype=torch.int32, device=DEV)
    at = torch.tensor(offs, dtype=torch.int64, device=DEV)
    tys = torch.tensor([TBE_TYPES[t] for t in _tbe_types(c)], dtype=torch.uint8, device=DEV)
    dim_offsets = torch.arange(T + 1, dtype=torch.int32, device=DEV) * D
    out = torch.empty((B, T * D), dtype=torch.float16 if c["out_fp16"] else torch.float32, device=DEV)
    status = ops.new_status(DEV)
    pooling = ops.EP_MEAN if c["mean_pooling"] else ops.EP_SUM
    return lambda: ops.int_nbit_split_embedding_bags(data, data, placements, at, tys, dim_offsets, T * D, indices, offsets,
                                                     pooling, indice_weights=iw, out=out, status=status)


def _prepare_fc(c, g):
    M, K, N, form = c["m"], c["k"], c["n"], c["form"]
    i8 = lambda *s: torch.randint(-127, 128, s, dtype=torch.int8, device=DEV, generator=g)
    status = ops.new_status(DEV)
    if form == "dynamic":
        x = torch.randn((M, K), device=DEV, generator=g).to(torch.float16)
        wt, bias = i8(N, K), torch.randn(N, device=DEV, generator=g)
        scales = torch.empty(N, device=DEV).uniform_(0.0005, 0.002, generator=g)
        offs = torch.zeros(N, dtype=torch.int32, device=DEV)
        if c["asym"]:
            offs.random_(-20, 21, generator=g)
        flags = 0 if c["asym"] else ops.FC_WEIGHT_OFFSETS_ZERO
        out = torch.empty((M, N), dtype=torch.float16, device=DEV)
        ws = torch.empty(ops.dynamic_fc_workspace_bytes(M, K, N), dtype=torch.uint8, device=DEV)
        return lambda: ops.dynamic_rowwise_quantized_fc(x, None, bias, scales, offs, weights_transposed=wt, flags=flags,
                                                        out=out, workspace=ws, status=status)
    x, out = i8(M, K), torch.empty((M, N), dtype=torch.int8, device=DEV)
    ws = torch.empty(max(8, ops.i8_gemm_workspace_bytes(M, K, N)), dtype=torch.uint8, device=DEV)
    in_scale, w_scale = 0.05, 0.01
    out_scale = in_scale * w_scale * 73 * 73 * math.sqrt(K) / 40   # results spread over the int8 range
    bias = torch.randint(-2 ** 16, 2 ** 16, (N,), dtype=torch.int32, device=DEV, generator=g)
    if form == "rowwise":
        w = i8(N, K)
        w_scales = torch.empty(N, device=DEV).uniform_(0.001, 0.02, generator=g).cpu().numpy()
        params = [torch.from_numpy(a).to(DEV) for a in
                  ops.rowwise_requant_params(w_scales, in_scale, np.float32(in_scale * w_scale), out_scale)]
        offs = torch.zeros(N, dtype=torch.int32, device=DEV)
        if c["asym"]:
            offs.random_(-20, 21, generator=g)
        flags = (0 if c["asym"] else ops.FC_WEIGHT_OFFSETS_ZERO) | (ops.FC_FUSE_RELU if c["relu"] else 0)
        sums = ops.i8_row_sums(w)
        return lambda: ops.rowwise_quantized_fc(x, w, bias, offs, params[:3], params[3:], 1, 3, 0, weights_row_sums=sums,
                                                flags=flags, out=out, workspace=ws, status=status)
    w = i8(K, N)
    w_off = 5 if c["asym"] else 0
    out_triple = ops.quantize_scale_offset_32to8(np.float32(in_scale * w_scale / out_scale))
    if form == "matmul":
        return lambda: ops.matmul_i8(x, w, 1, 3, w_off, out_triple, out=out, workspace=ws, status=status)
    bias_triple = ops.quantize_scale_offset_32to8(np.float32(1.0))
    return lambda: ops.fully_connected_i8(x, w, bias, 1, 3, w_off, 0, bias_triple, out_triple, out=out, workspace=ws,
                                          status=status)


def _graphed(call):
    """The call captured in a CUDA graph, as a server with fixed buffers keeps it."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            call()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side, capture_error_mode="thread_local"):
            out = call()
    torch.cuda.current_stream().wait_stream(side)

    def replay(held=call):   # the graph addresses what the call holds: weights, workspaces, inputs
        graph.replay()
        return out

    return replay


@functools.lru_cache(maxsize=1)
def _resnet_constants():
    layers = resnet.architecture()
    w = resnet.float_weights(layers)
    images = torch.randn((4, 3, 224, 224), generator=torch.Generator().manual_seed(7))
    _, ranges = resnet.float_forward(layers, w, images, DEV)
    return layers, resnet.quantize_network(layers, w, ranges)


def _prepare_resnet(c, g):
    model = resnet.ResNet50Int8(*_resnet_constants(), DEV)
    x = torch.randn((c["batch"], 3, c["size"], c["size"]), device=DEV, generator=g)
    call = lambda: model.forward(x)
    return _graphed(call) if c["graph"] else call


def _pooled_floats(table, dim, lengths, indices, bags):
    """The first `bags` bags of a uint8 table pooled in float, for calibration."""
    ln = lengths[:bags].long()
    start = torch.cumsum(ln, 0) - ln
    slot = torch.arange(int(ln.max()) + 1, device=DEV)[None]
    rows = table[indices[(start[:, None] + slot).clamp_(max=indices.shape[0] - 1)].long()]
    so = rows[..., dim:].contiguous().view(torch.float32)
    deq = rows[..., :dim].float() * so[..., :1] + so[..., 1:]
    return (deq * (slot < ln[:, None])[..., None]).sum(1)


def _recsys(c, g, tables, law):
    """The model of DLRMConfig's layers over `tables`, calibrated on a part of the request."""
    cfg = dlrm.DLRMConfig(tables=c["tables"], rows=c["rows"], dim=c["dim"], batch=c["batch"], bottom=(512, 256, c["dim"]),
                          mean_len=float(c["mean"]))
    dense = torch.randn((c["batch"], cfg.dense_in), device=DEV, generator=g)
    lengths = {t: _bag_lengths(c["batch"], c["mean"], law, g) for t in range(c["tables"])}
    indices = {t: _rows(max(1, int(lengths[t].sum())), c["rows"], law, True, g) for t in range(c["tables"])}
    few = min(64, c["batch"])
    pooled = torch.stack([_pooled_floats(tables[t], c["dim"], lengths[t], indices[t], few) for t in range(c["tables"])], 1)
    fm = dlrm.float_model(cfg)
    _, ranges = dlrm.float_forward(cfg, fm, dense[:few], pooled)
    return cfg, dense, lengths, indices, dlrm.quantize_model(cfg, fm, ranges)


def _prepare_dlrm(c, g):
    tables = {t: _fused_table(c["rows"], c["dim"], ops.UINT8_FUSED, g) for t in range(c["tables"])}
    cfg, dense, lengths, indices, qm = _recsys(c, g, tables, "power")
    model = dlrm.DLRMRank(cfg, qm, tables, device=DEV, exchange="local")
    bound = [model.prepare(lengths, indices, slab) for slab in range(2)]
    call = lambda: model.forward(dense, bound)
    return _graphed(call) if c["graph"] else call


def _prepare_request(c, g):
    T, B, D = c["tables"], c["batch"], c["dim"]
    tables = {t: _fused_table(c["rows"], D, ops.UINT8_FUSED, g) for t in range(T)}
    cfg, dense, lengths, indices, qm = _recsys(c, g, tables, "poisson")
    cap = B * c["mean"] * 3 // 2 + 64                     # indices a table's request may hold
    width = cfg.interaction_width
    f = runtime.Function("recsys")
    tabs = [f.static_placeholder("table%d" % t, c["rows"] * (D + 8)) for t in range(T)]
    p_x, p_idx = f.placeholder("dense", B * cfg.dense_in * 4), f.placeholder("indices", T * cap * 4)
    p_len, p_out = f.placeholder("lengths", T * B * 4), f.placeholder("scores", B * 4)
    ones, pooled, pool1 = f.activation("ones", cap * 4), f.activation("pooled", T * B * D * 4), f.activation("cat", T * B * D * 4)
    # SparseLengthsSum as it is lowered: weights of one; then Concat as it is lowered: InsertTensor per table
    f.splat(ones, n=cap, value=1.0)
    for t in range(T):
        f.frwq_slws((pooled, t * B * D * 4), tabs[t], ones, (p_idx, t * cap * 4), (p_len, t * B * 4), kind=ops.UINT8_FUSED,
                    rows=c["rows"], in_line=D + 8, out_line=D, segments=B, num_indices=cap, idx64=False)
    for t in range(T):
        f.insert_tensor(pool1, (pooled, t * B * D * 4), rows=B, width_bytes=D * 4, dest_pitch_bytes=T * D * 4,
                        dest_offset_bytes=t * D * 4)

    def mlp(part, x):
        for i, fc in enumerate(qm[part]):
            n, k = fc.w.shape
            pre = "%s%d_" % (part, i)
            y = f.activation(pre + "y", B * n)
            f.rowwise_fc(y, x, f.constant(pre + "w", fc.w), f.constant(pre + "s", fc.w_scales),
                         f.constant(pre + "o", fc.w_offsets), f.constant(pre + "b", fc.bias), M=B, K=k, N=n,
                         in_tqp=(fc.in_scale, fc.in_offset), bias_tqp=(fc.bias_scale, 0),
                         out_tqp=(fc.out_scale, fc.out_offset), relu=fc.relu)
            x = y
        return x, (fc.out_scale, fc.out_offset)

    xq, x0, inter = f.activation("xq", B * cfg.dense_in), f.activation("x0", B * D * 4), f.activation("inter", B * width)
    f.quantize(xq, p_x, n=B * cfg.dense_in, tqp=qm["dense_tqp"])
    last, tqp = mlp("bottom", xq)
    f.dequantize(x0, last, n=B * D, tqp=tqp)
    f.pairwise_dot(inter, x0, pool1, batch=B, tables=T, dim=D, quant=qm["interaction_tqp"])
    last, tqp = mlp("top", inter)
    f.dequantize(p_out, last, n=B, tqp=tqp)
    dm = runtime.DeviceManager(0).init()
    dm.add_network(f.compile())
    for t in range(T):
        at, nbytes = dm.placeholder_address("recsys", "table%d" % t)
        ops.device_tensor(at, (c["rows"], D + 8), torch.uint8).copy_(tables[t])
    io = {"dense": dm.io_buffer((B, cfg.dense_in), np.float32), "indices": dm.io_buffer((T, cap), np.int32),
          "lengths": dm.io_buffer((T, B), np.int32), "scores": dm.io_buffer((B, 1), np.float32)}
    io["dense"][:] = dense.cpu().numpy()
    io["indices"][:] = 0
    for t in range(T):
        ix = indices[t].cpu().numpy()[:cap]
        io["indices"][t, :ix.size] = ix
        io["lengths"][t] = lengths[t].cpu().numpy()
    torch.cuda.synchronize()

    def call():
        dm.run_function("recsys", io, outputs={"scores"})
        return io["scores"]

    return call


_PREPARE = {"pool": _prepare_pool, "tables": _prepare_tables, "tbe": _prepare_tbe, "fc": _prepare_fc,
            "resnet": _prepare_resnet, "dlrm": _prepare_dlrm, "request": _prepare_request}


def prepare(case, seed):
    return {"call": _PREPARE[case["path"]](case, _generator(seed))}


def run(state):
    return state["call"]()


# ------------------------------------------------------------------------------------------
# accounting
# ------------------------------------------------------------------------------------------
def _distinct(n, rows, law):
    """How many different rows n draws touch."""
    if law == "poisson":
        return rows * -math.expm1(-n / rows)
    at = np.exp(np.linspace(0.0, math.log(rows + 1.0), 4001))   # ranks, and the share of the draws below each
    share = (1 - at ** -0.05) / (1 - (rows + 1.0) ** -0.05)
    width = np.diff(at)
    return float(np.sum(width * -np.expm1(-n * np.diff(share) / width)))


def _pool_bytes(T, rows, bags, mean, law, line, dim, idx, weight, elem):
    """Each row that is touched once, indices and weights; lengths and results of the bags."""
    n = bags * mean
    return T * (_distinct(n, rows, law) * line + n * (idx + weight) + bags * (4 + dim * elem))


def work(case):
    c, path = case, case["path"]
    if path in ("pool", "tables"):
        kind, T = KINDS[c["kind"]], c.get("tables", 1)
        n = T * c["bags"] * c["mean"]
        elem = 2 if kind & 1 else 4
        return {"bytes": _pool_bytes(T, c["rows"], c["bags"], c["mean"], c.get("law", "poisson"),
                                     ops.fused_row_bytes(c["dim"], kind), c["dim"], 8 if c["idx64"] else 4, elem, elem),
                "flops": 2 * n * c["dim"]}
    if path == "tbe":
        D, idx = c["dim"], 8 if c["idx64"] else 4
        row = {"fp32": 4 * D, "fp16": 2 * D, "int8": D + 4, "int4": D // 2 + 4}
        return {"bytes": sum(_pool_bytes(1, c["rows"], c["bags"], c["mean"], "poisson", row[t], D, idx,
                                         4 if c["weighted"] else 0, 2 if c["out_fp16"] else 4) for t in _tbe_types(c)),
                "flops": 2 * c["tables"] * c["bags"] * c["mean"] * D}
    if path == "fc":
        M, K, N = c["m"], c["k"], c["n"]
        elem = 2 if c["form"] == "dynamic" else 1
        return {"bytes": elem * M * K + K * N + elem * M * N + 4 * N, "flops": 2 * M * K * N}
    if path == "resnet":
        layers = resnet.architecture()
        weights = sum(s["cin"] * s["cout"] * s["k"] ** 2 for l in layers if l[0] in ("conv", "block")
                      for s in ([l[1]] if l[0] == "conv" else l[2] + ([l[3]] if l[3] else []))) + 2048 * 1000
        return {"bytes": c["batch"] * (3 * c["size"] ** 2 + 1000) * 4 + weights,
                "flops": c["batch"] * resnet.conv_ops_per_image(layers, c["size"])}
    T, B, D = c["tables"], c["batch"], c["dim"]
    width = D + (T + 1) * T // 2
    macs = 256 * 512 + 512 * 256 + 256 * D + width * 1024 + 1024 * 1024 + 1024 * 512 + 512
    # pooled vectors need not leave the chip: their results are not counted
    law, idx = ("power", 8) if path == "dlrm" else ("poisson", 4)
    return {"bytes": _pool_bytes(T, c["rows"], B, c["mean"], law, D + 8, D, idx, 0, 0) + B * (256 + 1) * 4 + macs,
            "flops": B * (2 * macs + T * (T + 1) * D + 2 * T * c["mean"] * D)}


def tolerance(case):
    path = case["path"]
    if path in ("pool", "tables"):
        # fp32 sums in any order; an fp16 result is rounded once from such a sum
        return {"rel": 1e-3, "max": 4e-3} if KINDS[case["kind"]] & 1 else {"rel": 1e-5, "max": 1e-4}
    if path in ("dlrm", "request"):
        # int8 layers over fp32 sums of any order: now and then a value on the edge between two steps
        # of an int8 type falls the other way
        return {"rel": 5e-3, "max": 0.2}
    return "exact"   # defined bit for bit: integers, and running sums of a stated order and type
