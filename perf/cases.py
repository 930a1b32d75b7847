"""The calls whose speed counts: what a user of this framework has it do, through its public entry points.

The sizes are those of the benchmark configurations, the training presets and the tests: feature tables of up to a few million
rows, 32 to 400 columns (100, 110 and 200 among them), blocks of neighbour sampling with 1024 seeds and fan-outs of 5 to 15.
``listed`` holds one case for every kind of call, small ones among them; ``draw`` gives more cases of the same ranges.

Kinds:
  agg_sq, agg_vq, agg_two   the fused decode + mean aggregation of one sampled block (the first GraphSAGE layer)
  decode_sq, decode_vq      decompression of rows (the destination rows of a minibatch; a whole part of a table)
  encode_sq, encode_vq      the offline compressor: codebooks from a sample, then the codes of every row
  kmeans                    nearest centre of every sub-vector (codes of new features with given codebooks)
  minibatch                 the sampling loader: three hops of sampling and relabelling per minibatch
  train, infer              a whole training step (loader, forward, backward, Adam), and the forward pass alone
"""
import math

import torch
import torch.nn.functional as F

import F2CGTLib as capi
from f2cgt_b200 import compress, sage, synth
from f2cgt_b200.train_graphsage import DirectFusedAdam

DEGREE_EXPONENT = 2.1  # Zipf law of the synthetic graphs


def listed():
    return [
        # hot rows of one minibatch of 1024 seeds: the smallest call, latency only
        dict(name="decode_sq8_seeds", kind="decode_sq", rows=1024, dim=128, bits=8, slice=128),
        # part of a table decoded on the way to an uncompressed consumer: the longest stream
        dict(name="decode_vq_part", kind="decode_vq", rows=1_000_003, dim=128, slice=32, centers=256),
        # the 8-bit configuration: 10,000 rows of exactly 12 uniform neighbours
        dict(name="agg_sq8_uniform", kind="agg_sq", nodes=100_000, n_dst=10_000, fan=12, uniform=True, dim=128, bits=8, slice=128,
             index="int64", dropout=0.0),
        # the packed configuration, outermost block of 1024 seeds with fan-out 12,12,12
        dict(name="agg_sq4_block", kind="agg_sq", nodes=2_449_029, n_dst=59_000, fan=12, uniform=False, dim=128, bits=4, slice=128,
             index="int64", dropout=0.0),
        # a width that is no power of two (its column slice is rounded up to 8), int32 ids
        dict(name="agg_sq8_ragged", kind="agg_sq", nodes=2_449_029, n_dst=31_001, fan=12, uniform=False, dim=100, bits=8, slice=104,
             index="int32", dropout=0.0),
        # 16 subspaces of width 8
        dict(name="agg_vq_16x8", kind="agg_vq", nodes=2_449_029, n_dst=59_000, fan=12, uniform=False, dim=128, vq_slice=8, centers=256,
             index="int64", dropout=0.0),
        # two-level, 256 columns, fan-out 15, dropout on the aggregated rows
        dict(name="agg_two_256", kind="agg_two", nodes=2_449_029, n_dst=36_000, fan=15, uniform=False, dim=256, bits=4, slice=256, hot=0.02,
             vq_slice=64, centers=256, index="int64", dropout=0.5),
        # scalar compressor on a million rows, its codebook sample included
        dict(name="encode_sq4", kind="encode_sq", rows=1_000_000, dim=128, bits=4, slice=128),
        # vector compressor: k-means fits on a sample, then the codes of every row
        dict(name="encode_vq_32", kind="encode_vq", rows=400_000, dim=64, slice=32, centers=256),
        # k-means assignment of 8-dimensional sub-vectors
        dict(name="kmeans_8", kind="kmeans", rows=2_449_029, dim=8, centers=256, metric="cosine"),
        # one minibatch of the loader
        dict(name="minibatch_12_12_12", kind="minibatch", nodes=2_449_029, degree=50, batch=1024, fan1=12, fan2=12, fan3=12, index="int64"),
        # a training step of the "small" preset
        dict(name="train_step", kind="train", nodes=2_449_029, degree=50, batch=1024, fan1=12, fan2=12, fan3=12, index="int64", dim=128,
             hidden=128, classes=172, bits=8, hot=0.05, vq_slice=32, dropout=0.5, precision="tf32"),
    ]


KINDS = ("agg_sq", "agg_sq", "agg_vq", "agg_two", "decode_sq", "decode_vq", "encode_sq", "encode_vq", "kmeans", "minibatch", "train", "infer")
FANS = ((12, 12, 12), (15, 10, 5), (15, 15, 15), (10, 10, 5), (5, 5, 5))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, lo=32, hi=400):
    return rng.choice([64, 100, 110, 128, 128, 200, 256]) if rng.random() < 0.5 else rng.randint(lo, hi)


def _sq_slice(rng, dim):
    """The compressor's rule for one, two or four ranks: ceil(dim / ranks) rounded up to 8."""
    ranks = rng.choice([1, 1, 1, 2, 4])
    return ((dim + ranks - 1) // ranks + 7) // 8 * 8


def draw(rng):
    kind = rng.choice(KINDS)
    if kind.startswith("agg"):
        case = dict(kind=kind, nodes=_log(rng, 20_000, 2_500_000), n_dst=_log(rng, 200, 90_000), fan=rng.choice([5, 10, 12, 12, 15]),
                    uniform=rng.random() < 0.15, index=rng.choice(["int64", "int64", "int32"]), dropout=rng.choice([0.0, 0.0, 0.5]))
        if kind == "agg_sq":
            dim = _dim(rng)
            return dict(case, dim=dim, bits=rng.choice([1, 2, 4, 8, 8, 16]), slice=_sq_slice(rng, dim))
        if kind == "agg_vq":
            return dict(case, dim=_dim(rng, 32, 256), vq_slice=rng.choice([8, 16, 32, 64]), centers=rng.choice([256, 256, 256, 1024]))
        dim = rng.choice([64, 100, 128, 128, 256])
        return dict(case, dim=dim, bits=rng.choice([4, 8, 8]), slice=_sq_slice(rng, dim), hot=rng.uniform(0.01, 0.1),
                    vq_slice=rng.choice([8, 16, 32, 64]), centers=256)
    if kind == "decode_sq":
        dim = _dim(rng)
        return dict(kind=kind, rows=_log(rng, 256, 400_000), dim=dim, bits=rng.choice([1, 2, 4, 8, 8, 16]), slice=_sq_slice(rng, dim))
    if kind == "decode_vq":
        return dict(kind=kind, rows=_log(rng, 256, 400_000), dim=_dim(rng), slice=rng.choice([8, 16, 32, 64]), centers=rng.choice([256, 256, 1024]))
    if kind == "encode_sq":
        dim = _dim(rng, 32, 256)
        return dict(kind=kind, rows=_log(rng, 20_000, min(500_000, 72_000_000 // dim)), dim=dim, bits=rng.choice([1, 2, 4, 8, 16]), slice=_sq_slice(rng, dim))
    if kind == "encode_vq":
        width = rng.choice([8, 16, 32, 64])
        return dict(kind=kind, rows=_log(rng, 30_000, 400_000), dim=width * rng.randint(1, 2) - rng.choice([0, 0, 3]), slice=width,
                    centers=rng.choice([128, 256, 256]))
    if kind == "kmeans":
        dim = rng.choice([4, 8, 8, 16, 24, 32, 64])
        return dict(kind=kind, rows=_log(rng, 5_000, min(2_400_000, 68_000_000 // dim)), dim=dim, centers=rng.choice([100, 128, 256, 256]),
                    metric=rng.choice(["cosine", "cosine", "l2"]))
    fans = rng.choice(FANS)
    case = dict(kind=kind, nodes=_log(rng, 50_000, 2_449_029), degree=rng.randint(15, 50), batch=_log(rng, 64, 500 if fans == (15, 15, 15) else 1024), fan1=fans[0],
                fan2=fans[1], fan3=fans[2], index=rng.choice(["int64", "int64", "int32"]))
    if kind == "minibatch":
        return case
    return dict(case, dim=rng.choice([64, 100, 128, 128, 256]), hidden=rng.choice([64, 128, 128, 256]), classes=rng.randint(16, 172),
                bits=rng.choice([4, 8, 8]), hot=rng.uniform(0.01, 0.1), vq_slice=rng.choice([16, 32, 32, 64]), dropout=rng.choice([0.0, 0.5, 0.5]),
                precision=rng.choice(["tf32", "tf32", "tf32", "fp32", "bf16"]))


# ---------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _index_dtype(case):
    return torch.int32 if case["index"] == "int32" else torch.int64


def _block(case, g):
    """CSC of one sampled block: sources (and destinations) come up in proportion to their degree, as in neighbour sampling
    on a power-law graph, and a row keeps at most ``fan`` neighbours; uniform: every row has exactly ``fan``."""
    nodes, n_dst, fan, dt = case["nodes"], case["n_dst"], case["fan"], _index_dtype(case)
    if case["uniform"]:
        indptr = torch.arange(0, n_dst * fan + 1, fan, device="cuda")
        return indptr.to(dt), torch.randint(0, nodes, (n_dst * fan,), generator=g, device="cuda").to(dt)
    u = torch.rand(nodes, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-12)
    raw = u.pow(-1.0 / (DEGREE_EXPONENT - 1.0)).clamp_max(max(1.0, nodes / 20))
    deg = torch.floor(raw * (50.0 / raw.mean())).to(torch.int64)
    ends = torch.cumsum(deg, 0)

    def pick(n):
        return torch.searchsorted(ends, (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * ends[-1]).long(), right=True)

    indptr = torch.zeros(n_dst + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg[pick(n_dst)].clamp_max(fan), 0, out=indptr[1:])
    return indptr.to(dt), pick(int(indptr[-1])).to(dt)


def _sq_table(rows, dim, bits, width, g):
    """A table of random codes under codebooks made from a normal sample."""
    cb = synth.sq_codebook_from_sample(torch.randn(4096, dim, generator=g, device="cuda"), width)
    if bits == 16:
        return torch.randint(-32768, 32768, (rows, dim), generator=g, dtype=torch.int16, device="cuda"), cb
    return torch.randint(-128, 128, (rows, (dim * bits + 7) // 8), generator=g, dtype=torch.int8, device="cuda"), cb


def _vq_table(rows, dim, width, centers, g):
    n_cb = (dim + width - 1) // width
    dt = torch.uint8 if centers <= 256 else torch.int16
    return (torch.randint(0, centers, (rows, n_cb), generator=g, dtype=dt, device="cuda"),
            torch.randn(n_cb, centers, width, generator=g, device="cuda"))


def _manager(case, g):
    """The resident compressed table, as the trainer builds it."""
    nodes, dim = case["nodes"], case["dim"]
    if case["kind"] == "agg_sq":
        codes, cb = _sq_table(nodes, dim, case["bits"], case["slice"], g)
        return sage.CompressionManager(dim, ["sq"], [(case["slice"], case["bits"])], [cb], [codes])
    codes, cbs = _vq_table(nodes, dim, case["vq_slice"], case.get("centers", 256), g)
    if case["kind"] == "agg_vq":
        return sage.CompressionManager(dim, ["vq"], [(case["vq_slice"], -1)], [cbs], [codes])
    n_hot = max(1, int(nodes * case["hot"]))
    width = case.get("slice", (dim + 7) // 8 * 8)
    hot, cb = _sq_table(n_hot, dim, case["bits"], width, g)
    slot = torch.full((nodes,), -1, dtype=torch.int32, device="cuda")
    slot[torch.randperm(nodes, generator=g, device="cuda")[:n_hot]] = torch.arange(n_hot, dtype=torch.int32, device="cuda")
    return sage.CompressionManager(dim, ["sq", "vq"], [(width, case["bits"]), (case["vq_slice"], -1)], [cb, cbs], [hot, codes], slot)


def _features(case, g):
    """Rows around a few hundred prototypes, with noise: what a k-means codebook is for."""
    rows, dim = case["rows"], case["dim"]
    kinds = torch.randn(300, dim, generator=g, device="cuda")
    x = torch.randn(rows, dim, generator=g, device="cuda")
    return x.mul_(0.6).add_(kinds[torch.randint(0, 300, (rows,), generator=g, device="cuda")])


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    state = dict(case=case)
    if kind.startswith("agg"):
        state["manager"] = _manager(case, g)
        state["indptr"], state["indices"] = _block(case, g)
        state["dropout"] = dict(p=case["dropout"], seed=seed, offset=1, training=True) if case["dropout"] else None
    elif kind == "decode_sq":
        state["codes"], state["codebooks"] = _sq_table(case["rows"], case["dim"], case["bits"], case["slice"], g)
    elif kind == "decode_vq":
        state["codes"], state["codebooks"] = _vq_table(case["rows"], case["dim"], case["slice"], case["centers"], g)
    elif kind in ("encode_sq", "encode_vq"):
        state["features"], state["seed"] = _features(case, g), seed % 1000
    elif kind == "kmeans":
        state["x"] = torch.randn(case["rows"], case["dim"], generator=g, device="cuda")
        state["kmeans"] = capi.KMeans(torch.randn(case["centers"], case["dim"], generator=g, device="cuda"), case["metric"])
    else:
        indptr, indices = synth.power_law_graph(case["nodes"], case["degree"], DEGREE_EXPONENT, seed, "cuda", _index_dtype(case))
        ids = torch.randperm(case["nodes"], generator=g, device="cuda")[:120 * case["batch"]].to(_index_dtype(case))
        state["loader"] = sage.GPUSamplingDataloader(indptr, indices, ids, case["batch"], (case["fan1"], case["fan2"], case["fan3"]),
                                                     rng_seed=seed)
        state["batches"] = iter(state["loader"])
        if kind == "minibatch":
            state["flat"] = torch.zeros(_most_ids(case), dtype=_index_dtype(case), device="cuda")
        else:
            state["manager"] = _manager(case, g)
            state["labels"] = torch.randint(0, case["classes"], (case["nodes"],), generator=g, device="cuda")
            torch.manual_seed(seed)  # initial weights and dropout masks
            torch.backends.cuda.matmul.allow_tf32 = case["precision"] == "tf32"
            model = sage.SAGE(case["dim"], case["hidden"], case["classes"], 3, case["dropout"], state["manager"]).to("cuda")
            state["model"] = model.train(kind == "train")
            state["optimizer"] = DirectFusedAdam(model.parameters(), lr=0.003) if kind == "train" else None
            state["product"] = torch.bfloat16 if case["precision"] == "bf16" else None
    return state


# ---------------------------------------------------------------------------------------------- calls
def _next_batch(state):
    try:
        return next(state["batches"])
    except StopIteration:  # the epoch is over
        state["batches"] = iter(state["loader"])
        return next(state["batches"])


def _train(state):
    """One step of the training loop."""
    model, optimizer, loader = state["model"], state["optimizer"], state["loader"]
    _, output_nodes, blocks = _next_batch(state)
    y = state["labels"][output_nodes]
    with sage.products_in(state["product"]):
        pred = model(blocks)
    loss = F.cross_entropy(pred, y)
    loader.poke()
    optimizer.zero_grad(set_to_none=True)
    with sage.products_in(state["product"]):
        loss.backward()
    loader.poke()
    optimizer.step()
    loader.poke()
    return dict(loss=loss, pred=pred, grads=[p.grad for p in optimizer.params], params=optimizer.params, exp_avg=optimizer.exp_avg,
                exp_avg_sq=optimizer.exp_avg_sq)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind.startswith("agg"):
        return state["manager"].aggregate(state["indptr"], state["indices"], dropout=state["dropout"])
    if kind == "decode_sq":
        return capi.sq_decompress(state["codes"], state["codebooks"], case["bits"], case["slice"], case["dim"])
    if kind == "decode_vq":
        return capi.vq_decompress(state["codes"], state["codebooks"], case["dim"])
    if kind == "encode_sq":
        return compress.sq_compress_features(state["features"], case["bits"], case["slice"], seed=state["seed"])
    if kind == "encode_vq":
        return compress.vq_compress_features(state["features"], case["centers"], case["slice"], seed=state["seed"])
    if kind == "kmeans":
        return state["kmeans"].predict(state["x"])
    if kind == "train":
        return _train(state)
    input_nodes, output_nodes, blocks = _next_batch(state)
    if kind == "minibatch":
        # One tensor, since the sizes of the blocks differ from minibatch to minibatch (behind them it keeps what it held);
        # the index tensors carry a tail behind a block's edges that nothing reads.
        parts = [input_nodes, output_nodes]
        for b in blocks:
            parts += [b["indptr"], b["dst_nodes"], b["src_nodes"], b["indices_local"][:b["n_edges"]], b["indices_global"][:b["n_edges"]]]
        torch.cat(parts, out=state["flat"][:sum(t.numel() for t in parts)])
        return dict(flat=state["flat"], edges=[b["n_edges"] for b in blocks])
    with torch.no_grad(), sage.products_in(state["product"]):
        return state["model"](blocks)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _index_bytes(case):
    return 4 if case["index"] == "int32" else 8


def _codebook_bytes(case):
    return (case["dim"] + case["vq_slice"] - 1) // case["vq_slice"] * case.get("centers", 256) * case["vq_slice"] * 4


def _row_bytes(case):
    """Mean bytes of one compressed source row, slot lookup included (two-level: nodes are hot at random)."""
    dim = case["dim"]
    sq = (dim * case["bits"] + 7) // 8 if "bits" in case else 0
    if case["kind"] == "agg_sq":
        return sq
    vq = (dim + case["vq_slice"] - 1) // case["vq_slice"] * (1 if case.get("centers", 256) <= 256 else 2)
    return vq if case["kind"] == "agg_vq" else case["hot"] * sq + (1 - case["hot"]) * vq + 4


def _most_ids(case):
    """Upper bound of what one minibatch holds."""
    rows, total = case["batch"], case["batch"]
    for fan in (case["fan3"], case["fan2"], case["fan1"]):
        src = min(rows * (fan + 1), case["nodes"])
        total += 2 * rows * fan + 2 * rows + 1 + 2 * src
        rows = src
    return total


def _hops(case):
    """(destination rows, edges, source rows) of each block, innermost first; distinct sources are about 0.8 of the sampled
    edges in the first hop and half of them in the later ones."""
    rows, out = case["batch"], []
    for fan, distinct in ((case["fan3"], 0.8), (case["fan2"], 0.5), (case["fan1"], 0.45)):
        edges = rows * fan * 0.95
        src = min(rows + edges * distinct, case["nodes"])
        out.append((rows, edges, src))
        rows = int(src)
    return out


def work(case):
    kind, dim = case["kind"], case["dim"] if "dim" in case else 0
    if kind.startswith("agg"):
        edges = case["n_dst"] * case["fan"] * (1.0 if case["uniform"] else 0.97)
        ib = _index_bytes(case)
        books = 0 if kind == "agg_sq" else _codebook_bytes(case)
        return dict(bytes=edges * (ib + _row_bytes(case)) + case["n_dst"] * (ib + 4 * dim) + books, flops=edges * dim)
    if kind == "decode_sq":
        return dict(bytes=case["rows"] * ((dim * case["bits"] + 7) // 8 + 4 * dim), flops=0)
    if kind == "decode_vq":
        n_cb = (dim + case["slice"] - 1) // case["slice"]
        return dict(bytes=case["rows"] * (n_cb * (1 if case["centers"] <= 256 else 2) + 4 * dim) + n_cb * case["centers"] * case["slice"] * 4, flops=0)
    if kind == "encode_sq":
        sample = min(case["rows"], 250_000)
        return dict(bytes=case["rows"] * (4 * dim + (dim * case["bits"] + 7) // 8) + sample * 4 * dim, flops=0)
    if kind == "encode_vq":  # at least one iteration of each fit
        sample = min(case["rows"], 150_000)
        return dict(bytes=(case["rows"] + sample) * 4 * dim + case["rows"] * ((dim + case["slice"] - 1) // case["slice"]),
                    flops=2.0 * (case["rows"] + sample) * case["centers"] * dim)
    if kind == "kmeans":
        return dict(bytes=case["rows"] * (4 * dim + 8) + case["centers"] * 4 * dim, flops=2.0 * case["rows"] * case["centers"] * dim)
    ib, hops = _index_bytes(case), _hops(case)
    sampled = sum(rows * 3 * ib + edges * 3 * ib + src * ib for rows, edges, src in hops)
    if kind == "minibatch":
        return dict(bytes=sampled, flops=0)
    passes = 3 if kind == "train" else 1
    nbytes, flops = sampled + _codebook_bytes(case), 0.0
    widths = [(case["hidden"], case["classes"]), (case["hidden"], case["hidden"]), (dim, case["hidden"])]  # innermost hop = last layer
    for (rows, edges, src), (w_in, w_out), first in zip(hops, widths, (False, False, True)):
        if first:
            nbytes += edges * (ib + _row_bytes(case)) + rows * (_row_bytes(case) + 8 * dim + 4 * w_out)
            flops += (2 if kind == "train" else 1) * 4.0 * rows * w_in * w_out
        else:
            nbytes += passes * (src * 4 * w_in + edges * ib + rows * 4 * (w_in + w_out))
            flops += passes * 4.0 * rows * w_in * w_out
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    kind = case["kind"]
    if kind.startswith("agg"):
        return dict(rel=1e-5)  # fp32 sums of a few decoded rows
    if kind.startswith("decode"):
        return dict(rel=1e-6)
    if kind == "kmeans":
        return dict(rel=0.0, differ=1e-5)  # labels; equal distances
    if kind == "minibatch":
        return "exact"
    if kind == "encode_sq":
        return dict(rel=1e-5, differ=1e-5)  # statistics in fp32; codes on a quantisation boundary
    if kind == "encode_vq":
        return dict(rel=1e-3, max=0.1, differ=2e-3)  # centres in fp32 after several iterations, points between two centres
    # matrix products with tf32 (10 bits), bf16 (8 bits) or fp32 operands, then a step of Adam, whose update is the gradient's sign
    # where the gradient is small
    if kind == "infer":
        return dict(rel=dict(tf32=2e-3, bf16=1e-2, fp32=1e-5)[case["precision"]])
    return dict(rel=dict(tf32=5e-3, bf16=2e-2, fp32=3e-4)[case["precision"]], max=0.9)
