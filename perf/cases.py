"""Workloads of the framework's main paths, each as one call sequence that a user's program makes.

A case is a dict of plain values; ``kind`` names the path:

* ``dlrm``         one training step of the DLRM engine: pinned host batch in, tables and dense parameters updated;
* ``predict``      one inference call of the same engine (ranking requests: batches of some hundred to some thousand);
* ``mlp``          one Linear + ReLU layer of an MLP stack, forward and backward;
* ``bag``          pooled embedding lookup of a set of tables and the sparse optimizer on its gradients: one id per table
                   and sample (Criteo-like click logs), fixed multi-hot lists, or jagged weighted bags (``EmbeddingBag`` with
                   offsets and per-sample weights);
* ``interaction``  pairwise-dot feature interaction, forward and backward;
* ``table``        lookup + row-wise Adagrad (or SGD) update of a row-sharded table, storage dense;
* ``ps``           the parameter-server verbs on a hash-table shard: lookup, update, get;
* ``cache``        the GPU cache in front of a backing table: query, fetch and merge of the misses, update;
* ``kge``          one knowledge-graph embedding training step with chunked shared negatives.

Sizes are those of the repository's benchmark configurations (65,536 samples x 26 tables x 128, MLPs 13-512-256-128 and
479-1024-1024-512-256-1; the multi-hot list of the DCNv2 workload; 1,024 positives x 256 negatives x 400; 4,096 to 262,144
keys of 32 floats) and ragged ones between them.  Tables hold a million rows or two, so that a state can be built many times.
"""
from __future__ import annotations

import math

import torch

from recstore_b200.cache.gpu_cache import GpuCache, merge_op
from recstore_b200.models.dlrm import DLRM, DLRMConfig
from recstore_b200.models.kge import KGEConfig, KGEModel
from recstore_b200.ops import functional as F_
from recstore_b200.parallel.peer import PeerContext
from recstore_b200.parallel.sharded_table import ShardedEmbeddingTable
from recstore_b200.utils.data import loguniform_table_rows, spread_permutation, zipf_from_uniform

BOT, TOP = (512, 256, 128), (1024, 1024, 512, 256, 1)
MULTIHOT = "3,2,1,2,6,1,1,1,1,7,3,8,1,6,9,5,1,1,1,12,100,27,10,3,1,1"
LR, EPS = 0.01, 1e-10


def listed():
    return [
        # the headline workload: 65,536 samples on one GPU, 26 tables, Zipf 1.2 ids, pinned host batches, double buffered
        {"name": "dlrm_train_65536", "kind": "dlrm", "batch": 65536, "tables": 26, "rows": 2000000, "alpha": 1.2},
        # a ranking request: some hundred candidates scored by the same model
        {"name": "predict_1000", "kind": "predict", "batch": 1000, "tables": 26, "rows": 2000000, "alpha": 1.2},
        # the widest layer of the top MLP at the headline batch
        {"name": "mlp_65536_1024_1024", "kind": "mlp", "m": 65536, "n": 1024, "k": 1024},
        # the sparse side of the headline workload by itself: one id per table and sample, gradient norms at hand
        {"name": "bag_onehot_65536", "kind": "bag", "batch": 65536, "tables": 26, "dim": 128, "rows": 2000000, "alpha": 1.2,
         "bags": "one", "optimizer": "rowwise_adagrad", "norms": True},
        # the multi-hot workload: one eighth of its global batch, 214 ids per sample, one list of 100
        {"name": "bag_multihot_8192", "kind": "bag", "batch": 8192, "tables": 26, "dim": 128, "rows": 2000000, "alpha": 1.1,
         "bags": "multi", "optimizer": "rowwise_adagrad", "norms": True},
        # a small EmbeddingBag layer: jagged weighted bags, some of them empty, narrow rows, SGD
        {"name": "bag_jagged_500", "kind": "bag", "batch": 500, "tables": 5, "dim": 32, "rows": 50000, "alpha": 1.05,
         "bags": "jagged", "optimizer": "sgd", "norms": False},
        # the interaction of the headline workload by itself
        {"name": "interaction_65536", "kind": "interaction", "batch": 65536, "features": 27, "dim": 128},
        # the parameter-server micro-benchmark's largest batch, dense storage
        {"name": "table_262144_d32", "kind": "table", "keys": 262144, "dim": 32, "rows": 4000000, "alpha": 1.1,
         "optimizer": "rowwise_adagrad"},
        # an ordinary batch of the same on a hash-table shard with arbitrary 64-bit keys
        {"name": "ps_32768_d32", "kind": "ps", "keys": 32768, "dim": 32, "rows": 1000000, "alpha": 0.9},
        # cached embeddings: a deduplicated batch against a cache that holds about three quarters of it
        {"name": "cache_65536_d32", "kind": "cache", "keys": 65536, "dim": 32, "items": 400000, "space": 4000000, "alpha": 0.9},
        # knowledge-graph training at its benchmark shape: a model scored by cross products, and one scored pair by pair
        {"name": "kge_transe_1024", "kind": "kge", "model": "TransE_l2", "batch": 1024, "chunk": 256, "negs": 256, "dim": 400,
         "entities": 200000, "graph": True},
        {"name": "kge_rotate_1024", "kind": "kge", "model": "RotatE", "batch": 1024, "chunk": 256, "negs": 256, "dim": 400,
         "entities": 200000, "graph": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dlrm", "predict", "mlp", "mlp", "bag", "bag", "interaction", "table", "table", "ps", "cache", "kge", "kge"])
    if kind == "dlrm":
        return {"kind": kind, "batch": _log(rng, 500, 65536), "tables": rng.randint(3, 26), "rows": _log(rng, 20000, 2000000),
                "alpha": rng.choice([0.9, 1.05, 1.2])}
    if kind == "predict":
        return {"kind": kind, "batch": _log(rng, 50, 20000), "tables": rng.randint(3, 26), "rows": _log(rng, 20000, 2000000),
                "alpha": rng.choice([0.9, 1.05, 1.2])}
    if kind == "mlp":
        return {"kind": kind, "m": _log(rng, 130, 65536), "n": rng.choice([128, 256, 512, 1024]), "k": rng.choice([64, 128, 256, 512, 1024])}
    if kind == "bag":
        bags = rng.choice(["one", "multi", "jagged"])
        return {"kind": kind, "batch": _log(rng, 100, 8192 if bags == "multi" else 65536 if bags == "one" else 16384), "tables": rng.randint(1, 26),
                "dim": rng.choice([16, 32, 64, 100, 128, 256]) if bags != "multi" else 128, "rows": _log(rng, 5000, 1000000),
                "alpha": rng.choice([0.9, 1.05, 1.1, 1.2]), "bags": bags, "optimizer": rng.choice(["rowwise_adagrad", "rowwise_adagrad", "sgd"]),
                "norms": rng.random() < 0.5}
    if kind == "interaction":
        return {"kind": kind, "batch": _log(rng, 100, 65536), "features": rng.randint(3, 32), "dim": rng.choice([16, 32, 64, 128])}
    if kind == "table":
        dim = rng.choice([16, 32, 64, 100, 128, 400])
        return {"kind": kind, "keys": _log(rng, 1000, 262144 if dim <= 64 else 65536), "dim": dim, "rows": _log(rng, 50000, 1000000),
                "alpha": rng.choice([0.9, 1.1, 1.3]), "optimizer": rng.choice(["rowwise_adagrad", "rowwise_adagrad", "sgd"])}
    if kind == "ps":
        return {"kind": kind, "keys": _log(rng, 1000, 131072), "dim": rng.choice([16, 32, 64, 128]), "rows": _log(rng, 50000, 1000000),
                "alpha": rng.choice([0.9, 1.1, 1.3])}
    if kind == "cache":
        return {"kind": kind, "keys": _log(rng, 1000, 262144), "dim": rng.choice([16, 32, 64, 128]), "items": _log(rng, 100000, 1000000),
                "space": 4000000, "alpha": rng.choice([0.9, 1.1])}
    chunk = rng.choice([64, 128, 256])
    return {"kind": "kge", "model": rng.choice(["TransE_l2", "DistMult", "ComplEx", "SimplE", "TransE_l1", "RotatE"]),
            "batch": chunk * rng.randint(1, 1024 // chunk), "chunk": chunk, "negs": rng.choice([16, 64, 128, 256]),
            "dim": rng.choice([64, 120, 200, 400]), "entities": _log(rng, 20000, 200000), "graph": rng.random() < 0.7}


class _State:
    """What one case keeps between calls; the exchange windows of its context go back when it does."""

    ctx = None

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        ctx, self.ctx = self.ctx, None
        if ctx is not None:
            ctx.free_all()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g)


def _zipf(g, n, rows, alpha):
    return zipf_from_uniform(torch.rand(n, device="cuda", dtype=torch.float64, generator=g), rows, alpha)


def _spread(ids, rows):
    """Popular ids anywhere in the table."""
    a, b = spread_permutation(rows)
    return (ids * a + b) % rows


def _rows_of(case):
    return loguniform_table_rows(case["tables"], 10, max(100, case["rows"] // 3), case["rows"], 7)


# ---------------------------------------------------------------------------------------------- inputs
def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s.kind = case["kind"]
    return s


def _prepare_dlrm(case, seed):
    rows, B = _rows_of(case), case["batch"]
    eng = DLRM(DLRMConfig(table_rows=rows, batch=B, seed=seed, bottom_mlp=BOT, top_mlp=TOP))
    g = _gen(seed)
    dense = torch.log1p(torch.empty(B, 13, device="cuda").exponential_(1.0, generator=g))
    labels = (torch.rand(B, device="cuda", generator=g) < 0.25).float()
    ids = [_zipf(g, B, n, case["alpha"]).cpu() for n in rows]
    return _State(ctx=eng.ctx, eng=eng, batch=eng.make_pinned_batch(dense.cpu(), ids, labels.cpu()), last=None)


def _prepare_mlp(case, seed):
    g, (M, N, K) = _gen(seed), (case["m"], case["n"], case["k"])
    w = (_randn(g, N, K) * math.sqrt(2.0 / (N + K))).bfloat16()
    e = dict(device="cuda")
    return _State(x=torch.relu(_randn(g, M, K)).bfloat16(), dy=(_randn(g, M, N) / M).bfloat16(), w=w, wt=w.t().contiguous(), b=_randn(g, N) * 0.1,
                  y=torch.empty(M, N, dtype=torch.bfloat16, **e), dx=torch.empty(M, K, dtype=torch.bfloat16, **e), gw=torch.zeros(N, K, **e),
                  gb=torch.zeros(N, **e), status=torch.zeros(1, dtype=torch.int64, **e))


def _prepare_bag(case, seed):
    g, (B, T, D) = _gen(seed), (case["batch"], case["tables"], case["dim"])
    rows = _rows_of(case)
    i64, i32 = dict(dtype=torch.int64, device="cuda"), dict(dtype=torch.int32, device="cuda")
    base = [0]
    for n in rows:
        base.append(base[-1] + n)
    s = _State(B=B, T=T, D=D, rows=rows, weight=torch.empty(base[-1], D, device="cuda").uniform_(-0.05, 0.05, generator=g), offsets=None, psw=None,
               hot=None, hot_base=None)
    s.state = torch.zeros(base[-1], device="cuda") if case["optimizer"] == "rowwise_adagrad" else None
    s.table_base, s.table_rows = torch.tensor(base[:-1], **i64), torch.tensor(rows, **i64)
    if case["bags"] == "jagged":
        lens = torch.randint(0, 9, (T * B,), device="cuda", generator=g)
        s.offsets = torch.cat([torch.zeros(1, **i64), lens.cumsum(0)])
        counts = lens.view(T, B).sum(1).tolist()
    else:
        hot = [1] * T if case["bags"] == "one" else [int(h) for h in MULTIHOT.split(",")][:T]
        s.hot, counts = torch.tensor(hot, **i32), [h * B for h in hot]
        lens = s.hot.long().repeat_interleave(B)
        s.hot_base = torch.tensor([sum(counts[:t]) for t in range(T)], **i64)
    s.bag_of = torch.repeat_interleave(torch.arange(T * B, device="cuda"), lens)
    s.ids = torch.cat([_zipf(g, max(c, 0), n, case["alpha"]) for c, n in zip(counts, rows)])
    s.nnz = s.ids.numel()
    if case["bags"] == "jagged":
        s.psw = torch.rand(s.nnz, device="cuda", generator=g) + 0.5
    s.out = torch.empty(B, T * D, dtype=torch.bfloat16, device="cuda")
    s.dst, s.col = torch.tensor([s.out.data_ptr()], **i64), torch.arange(T, **i32) * D
    s.row_idx, s.occ2bag = torch.empty(max(s.nnz, 1), **i64), torch.empty(max(s.nnz, 1), **i32)
    s.grad = (_randn(g, B, T * D) * 0.01).bfloat16()
    s.gnorm = s.grad.float().view(B, T, D).pow(2).sum(-1).contiguous() if case["norms"] and s.state is not None else None
    s.status = torch.zeros(1, **i64)
    return s


def _prepare_interaction(case, seed):
    g, (B, F, D) = _gen(seed), (case["batch"], case["features"], case["dim"])
    bf = dict(dtype=torch.bfloat16, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    ld = (D + F * (F - 1) // 2 + 63) // 64 * 64
    t = _randn(g, B, F, D) * 0.3
    t[:, 0].relu_()
    s = _State(B=B, F=F, D=D, T=t.bfloat16(), out=torch.empty(B, ld, **bf), dout=(_randn(g, B, ld) * 0.1).bfloat16(), dx=torch.empty(B, D, **bf),
               G=torch.empty(B, (F - 1) * D, **bf), norms=torch.empty(B, F - 1, device="cuda"), owner=torch.zeros(F - 1, **i32),
               gcol=torch.arange(F - 1, **i32) * D)
    s.gt = torch.tensor([s.G.data_ptr()], dtype=torch.int64, device="cuda")
    s.nt = torch.tensor([s.norms.data_ptr()], dtype=torch.int64, device="cuda")
    return s


def _prepare_table(case, seed):
    g, (n, D, N) = _gen(seed), (case["keys"], case["dim"], case["rows"])
    ctx = PeerContext(0, 1)
    init = torch.empty(N, D, device="cuda").uniform_(-0.05, 0.05, generator=g)
    t = ShardedEmbeddingTable(ctx, "rows", N, D, max_keys=n, lr=LR, eps=EPS, optimizer=case["optimizer"], init=init)
    return _State(ctx=ctx, t=t, ids=_spread(_zipf(g, n, N, case["alpha"]), N), grad=_randn(g, n, D) * 0.01)


def _prepare_ps(case, seed):
    g, (n, D, N) = _gen(seed), (case["keys"], case["dim"], case["rows"])
    ctx = PeerContext(0, 1)
    t = ShardedEmbeddingTable(ctx, "rows", N, D, max_keys=n, lr=LR, eps=EPS, hashed=True)
    key = lambda i: (i + 1) * 2654435761 + 12345                                     # noqa: E731  keys are not row numbers
    first = torch.empty(N, D, device="cuda").uniform_(-0.05, 0.05, generator=g)
    for k in range(0, N, n):
        part = torch.arange(k, min(N, k + n), device="cuda")
        t.put(key(part), first[k:k + n])
    rank = _spread(_zipf(g, n, N, case["alpha"]), N)
    return _State(ctx=ctx, t=t, ids=key(rank), rank=rank, first=first, grad=_randn(g, n, D) * 0.01)


def _prepare_cache(case, seed):
    g, (n, D) = _gen(seed), (case["keys"], case["dim"])
    back = _randn(g, case["space"], D) * 0.05
    perm = torch.randperm(case["space"], device="cuda", generator=g)
    cache = GpuCache(case["items"], D, "cuda:0")
    warm = perm[:case["items"] * 3 // 4]
    for k in range(0, warm.numel(), 1 << 17):
        cache.Replace(warm[k:k + (1 << 17)], back[warm[k:k + (1 << 17)]])
    keys = torch.unique(perm[_zipf(g, 4 * n, case["space"], case["alpha"])])
    keys = keys[torch.randperm(keys.numel(), device="cuda", generator=g)][:n].contiguous()
    return _State(cache=cache, back=back, keys=keys, values=torch.empty(keys.numel(), D, device="cuda"))


def _prepare_kge(case, seed):
    g, bs, N = _gen(seed), case["batch"], case["entities"]
    ctx = PeerContext(0, 1)
    m = KGEModel(KGEConfig(n_entities=N, n_relations=1000, dim=case["dim"], model=case["model"], batch=bs, neg_chunk_size=case["chunk"],
                           neg_sample_size=case["negs"], seed=seed, use_cuda_graph=case["graph"]), ctx)
    pick = lambda n, hi: torch.randint(0, hi, (n,), device="cuda", generator=g)      # noqa: E731
    h, t = (_spread(_zipf(g, bs, N, 1.3), N) for _ in range(2))
    return _State(ctx=ctx, m=m, h=h, r=pick(bs, 1000), t=t, neg=pick(bs // case["chunk"] * case["negs"], N))


_PREPARE = {"dlrm": _prepare_dlrm, "predict": _prepare_dlrm, "mlp": _prepare_mlp, "bag": _prepare_bag, "interaction": _prepare_interaction,
            "table": _prepare_table, "ps": _prepare_ps, "cache": _prepare_cache, "kge": _prepare_kge}


# ---------------------------------------------------------------------------------------------- one pass
def run(s):
    return _RUN[s.kind](s)


def _run_dlrm(s):
    # the double-buffered loop: submit a batch, then read the loss of the one before
    h = s.eng.submit(s.batch)
    loss = s.last.result() if s.last is not None else 0.0
    s.last = h
    return {"loss_before": loss, "dense": s.eng.master, "rows": s.eng.weight, "state": s.eng.state}


def _run_predict(s):
    return {"prob": s.eng.predict(s.batch)}


def _run_mlp(s):
    F_.gemm_bf16(s.x, s.w, s.y, epi=F_.EPI_RELU, bias=s.b, status=s.status)
    s.gw.zero_()
    s.gb.zero_()
    F_.colsum_bf16(s.dy, s.gb)
    F_.gemm_bf16(s.dy, s.x, s.gw, mode=1, epi=F_.EPI_ATOMIC_F32, status=s.status)
    F_.gemm_bf16(s.dy, s.wt, s.dx, epi=F_.EPI_RELU_MASK, aux=s.x, status=s.status)
    return {"y": s.y, "dx": s.dx, "gw": s.gw, "gb": s.gb}


def _run_bag(s):
    F_.emb_forward(s.weight, s.table_base, s.table_rows, s.ids, offsets=s.offsets, hotness=s.hot, hot_base=s.hot_base, per_sample_weights=s.psw,
                   T=s.T, B=s.B, D=s.D, B_local=s.B, dst_table=s.dst, dst_row_stride=s.T * s.D, dst_col=s.col, row_idx=s.row_idx,
                   occ2bag=s.occ2bag, status=s.status)
    F_.emb_backward(s.weight, s.state, s.row_idx, s.occ2bag, s.nnz, s.grad, grad_col=s.col, grad_row_stride=s.T * s.D, B=s.B, D=s.D,
                    per_sample_weights=s.psw, lr=LR, eps=EPS, optimizer="sgd" if s.state is None else "rowwise_adagrad", status=s.status,
                    gnorm=s.gnorm, gnorm_stride=s.T if s.gnorm is not None else 0)
    return {"pooled": s.out, "rows": s.weight, "state": s.state}


def _run_interaction(s):
    F_.interaction_forward(s.T, s.B, s.F, s.D, s.out)
    F_.interaction_backward(s.T, s.dout, s.B, s.F, s.D, s.dx, s.gt, s.owner, s.gcol, s.G.stride(0), 0, True, s.nt, s.F - 1)
    return {"out": s.out, "dx": s.dx, "grads": s.G, "norms": s.norms}


def _run_table(s):
    rows = s.t.lookup(s.ids)
    s.t.update(s.grad)
    return {"rows": rows, "weight": s.t.weight, "state": s.t.state}


def _run_ps(s):
    rows = s.t.lookup(s.ids)
    s.t.update(s.grad)
    after, found = s.t.get(s.ids)
    return {"rows": rows, "after": after, "found": found}


def _run_cache(s):
    r = s.cache.Query(s.keys, s.values)
    merge_op(r.values, s.back[r.missing_keys], r.missing_index)
    s.cache.Update(s.keys, r.values)
    return {"values": r.values}


def _run_kge(s):
    loss = s.m.train_step(s.h, s.r, s.t, s.neg)
    return {"loss": loss, "entities": s.m.entity.weight, "entity_state": s.m.entity.state, "relations": s.m.relation.weight,
            "relation_state": s.m.relation.state}


_RUN = {"dlrm": _run_dlrm, "predict": _run_predict, "mlp": _run_mlp, "bag": _run_bag, "interaction": _run_interaction, "table": _run_table,
        "ps": _run_ps, "cache": _run_cache, "kge": _run_kge}


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _distinct(n, rows, alpha):
    """Expected number of distinct ids among n Zipf draws of a table."""
    k = torch.arange(rows, dtype=torch.float64)
    edge = (k + 1.0) ** (1.0 - alpha)
    p = (edge - (k + 2.0) ** (1.0 - alpha)) / (1.0 - (rows + 1.0) ** (1.0 - alpha))
    return float((1.0 - torch.exp(n * torch.log1p(-p.clamp(max=1.0 - 1e-12)))).sum())


def _layers(case):
    F = case["tables"] + 1
    widths = [13] + list(BOT)
    top = [128 + F * (F - 1) // 2] + list(TOP)
    return list(zip(widths[:-1], widths[1:])) + list(zip(top[:-1], top[1:]))


def work(case):
    kind = case["kind"]
    if kind in ("dlrm", "predict"):
        B, T, D = case["batch"], case["tables"], 128
        distinct = sum(_distinct(B, n, case["alpha"]) for n in _rows_of(case))
        macs, par = sum(k * n for k, n in _layers(case)), sum(k * n + n for k, n in _layers(case))
        io = B * (13 * 4 + T * 8 + 4)
        if kind == "predict":
            return {"bytes": io + distinct * D * 4 + par * 4, "flops": 2.0 * B * (macs + (T + 1) ** 2 * D / 2)}
        return {"bytes": io + distinct * (D * 4 * 2 + 8) + par * 8, "flops": 6.0 * B * (macs + (T + 1) ** 2 * D / 2)}
    if kind == "mlp":
        M, N, K = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (2 * M * K + 2 * M * N + 2 * N * K) + 4 * (N * K + 2 * N), "flops": 6.0 * M * N * K}
    if kind == "bag":
        B, T, D, rows = case["batch"], case["tables"], case["dim"], _rows_of(case)
        hot = {"one": [1.0] * T, "jagged": [4.0] * T, "multi": [float(h) for h in MULTIHOT.split(",")][:T]}[case["bags"]]
        ids = sum(hot) * B
        distinct = sum(_distinct(h * B, n, case["alpha"]) for h, n in zip(hot, rows))
        extra = 8 if case["optimizer"] == "rowwise_adagrad" else 0
        return {"bytes": ids * 8 + distinct * (D * 8 + extra) + 2 * B * T * D * 2, "flops": 4.0 * ids * D}
    if kind == "interaction":
        B, F, D = case["batch"], case["features"], case["dim"]
        z = D + F * (F - 1) // 2
        return {"bytes": B * (2 * F * D * 2 + 2 * z * 2 + (F - 1) * 4), "flops": 3.0 * B * F * F * D}
    if kind in ("table", "ps"):
        n, D = case["keys"], case["dim"]
        distinct = _distinct(n, case["rows"], case["alpha"])
        return {"bytes": n * (8 + (3 if kind == "ps" else 2) * D * 4) + distinct * D * 8, "flops": 4.0 * n * D}
    if kind == "cache":
        n, D = case["keys"], case["dim"]
        return {"bytes": n * (8 + 256 + 4 * D * 4), "flops": 0.0}
    bs, D, neg = case["batch"], case["dim"], case["batch"] // case["chunk"] * case["negs"]
    return {"bytes": (2 * bs + neg + bs) * D * 4 * 2.0, "flops": 6.0 * bs * case["negs"] * D}


def tolerance(case):
    kind = case["kind"]
    # bf16 activations and gradients through seven GEMMs each way: a differing rounding in one layer travels on; the
    # accumulators hold squares of gradients
    if kind == "dlrm":
        return {"rel": 0.02, "max": 0.9}
    if kind == "predict":
        return {"rel": 0.01, "max": 0.2}
    if kind in ("mlp", "interaction"):
        return {"rel": 0.004, "max": 0.1}                    # bf16 results
    if kind == "bag":
        return {"rel": 0.004, "max": 0.1}                    # bf16 pooled rows; fp32 rows and accumulators
    if kind == "table" or kind == "ps":
        return {"rel": 1e-5, "max": 1e-3}                    # fp32 sums in any order
    if kind == "cache":
        return "exact"                                       # rows are copied
    if case["model"] in ("RotatE", "TransE_l1"):
        return {"rel": 1e-3, "max": 0.5}                     # fp32, with signs and directions of near-zero differences
    return {"rel": 0.005, "max": 0.9}                        # bf16 cross products


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    s = prepare(case, seed)
    with torch.no_grad():
        return _EXACT[case["kind"]](case, s)


def _adagrad(weight, state, idx, grad, lr, eps, norm=None):
    w, st = weight.double(), state.double()
    st.index_add_(0, idx, grad.pow(2).mean(1) if norm is None else norm)
    w.index_add_(0, idx, -lr * grad / (st[idx].sqrt() + eps).unsqueeze(1))
    return w, st


def _exact_forward(s, p, rows):
    """Probabilities and logits of the model with parameters ``p`` on the pooled rows ``rows`` [T, B, D]."""
    x = s.batch.dense.cuda().double()
    for i in range(len(BOT)):
        x = torch.relu(x @ p[f"bot.{i}.weight"].t() + p[f"bot.{i}.bias"])
    t = torch.cat([x.unsqueeze(1), rows.transpose(0, 1)], 1)
    li, lj = torch.tril_indices(t.shape[1], t.shape[1], offset=-1, device="cuda")
    z = torch.cat([x, torch.bmm(t, t.transpose(1, 2))[:, li, lj]], 1)
    for i in range(len(TOP) - 1):
        z = torch.relu(z @ p[f"top.{i}.weight"].t() + p[f"top.{i}.bias"])
    return z @ p["head.weight"] + p["head.bias"]


def _exact_dlrm(case, s):
    e, T, B = s.eng, case["tables"], case["batch"]
    ids = s.batch.ids.cuda().view(T, B) + e.table_base.view(T, 1)
    p = {k: v.double() for k, v in e.dense_state().items()}
    rows = e.weight[ids].double()
    if case["kind"] == "predict":
        return {"prob": torch.sigmoid(_exact_forward(s, p, rows))}
    with torch.enable_grad():
        p = {k: v.requires_grad_(True) for k, v in p.items()}
        rows.requires_grad_(True)
        y = s.batch.labels.cuda().double()
        torch.nn.functional.binary_cross_entropy_with_logits(_exact_forward(s, p, rows), y).backward()
    w, st = _adagrad(e.weight, e.state, ids.reshape(-1), rows.grad.reshape(T * B, -1), e.cfg.emb_lr, e.cfg.emb_eps)
    master = e.master.double()
    e.load_dense_state({k: v.grad.float() for k, v in p.items()})        # the gradients in the parameters' own layout
    return {"loss_before": None, "dense": master - e.cfg.mlp_lr * e.master.double(), "rows": w, "state": st}


def _exact_mlp(case, s):
    x, dy, w = s.x.double(), s.dy.double(), s.w.double()
    return {"y": torch.relu(x @ w.t() + s.b.double()), "dx": (dy @ w) * (x > 0), "gw": dy.t() @ x, "gb": dy.sum(0)}


def _exact_bag(case, s):
    B, T, D = s.B, s.T, s.D
    rows = s.ids + s.table_base[s.bag_of // B]
    w = s.psw.double() if s.psw is not None else torch.ones(s.nnz, dtype=torch.float64, device="cuda")
    pooled = torch.zeros(T * B, D, dtype=torch.float64, device="cuda").index_add_(0, s.bag_of, s.weight[rows].double() * w.unsqueeze(1))
    g = s.grad.view(B, T, D).transpose(0, 1).reshape(T * B, D)[s.bag_of].double() * w.unsqueeze(1)
    out = {"pooled": pooled.view(T, B, D).transpose(0, 1).reshape(B, T * D), "state": None}
    if s.state is None:
        out["rows"] = s.weight.double().index_add_(0, rows, -LR * g)
    else:
        out["rows"], out["state"] = _adagrad(s.weight, s.state, rows, g, LR, EPS)
    return out


def _exact_interaction(case, s):
    t, D, F, B = s.T.double(), s.D, s.F, s.B
    li, lj = torch.tril_indices(F, F, offset=-1, device="cuda")
    out = torch.zeros(B, s.out.shape[1], dtype=torch.float64, device="cuda")
    out[:, :D] = t[:, 0]
    out[:, D:D + li.numel()] = torch.bmm(t, t.transpose(1, 2))[:, li, lj]
    dz = torch.zeros(B, F, F, dtype=torch.float64, device="cuda")
    dz[:, li, lj] = s.dout[:, D:D + li.numel()].double()
    dt = torch.bmm(dz + dz.transpose(1, 2), t)
    dx = (dt[:, 0] + s.dout[:, :D].double()) * (t[:, 0] > 0)
    return {"out": out, "dx": dx, "grads": dt[:, 1:].reshape(B, -1), "norms": dt[:, 1:].pow(2).sum(-1)}


def _exact_table(case, s):
    g, w = s.grad.double(), s.t.weight
    rows = w[s.ids].double()
    if s.t.state is None:
        return {"rows": rows, "weight": w.double().index_add_(0, s.ids, -LR * g), "state": None}
    weight, state = _adagrad(w, s.t.state, s.ids, g, LR, EPS)
    return {"rows": rows, "weight": weight, "state": state}


def _exact_ps(case, s):
    w, _ = _adagrad(s.first, torch.zeros(case["rows"], device="cuda"), s.rank, s.grad.double(), LR, EPS)
    return {"rows": s.first[s.rank].double(), "after": w[s.rank], "found": None}


def _exact_cache(case, s):
    return {"values": s.back[s.keys].double()}


def _exact_kge(case, s):
    m, name, D, bs = s.m, case["model"], case["dim"], case["batch"]
    cs, ns, H = case["chunk"], case["negs"], case["dim"] // 2
    with torch.enable_grad():
        h, t, neg = (m.entity.weight[i].double().requires_grad_(True) for i in (s.h, s.t, s.neg))
        r = m.relation.weight[s.r].double().requires_grad_(True)

        def score(hh, rr, tt):
            if name == "TransE_l2":
                return m.cfg.gamma - (hh + rr - tt).norm(dim=-1)
            if name == "TransE_l1":
                return m.cfg.gamma - (hh + rr - tt).abs().sum(-1)
            if name == "DistMult":
                return (hh * rr * tt).sum(-1)
            h0, h1, t0, t1 = hh[..., :H], hh[..., H:], tt[..., :H], tt[..., H:]
            if name == "ComplEx":
                r0, r1 = rr[..., :H], rr[..., H:]
                return (h0 * t0 * r0 + h1 * t1 * r0 + h0 * t1 * r1 - h1 * t0 * r1).sum(-1)
            if name == "SimplE":
                return (0.5 * (h0 * rr[..., :H] * t1 + t0 * rr[..., H:] * h1).sum(-1)).clamp(-20, 20)
            ph = rr * (math.pi / m.emb_init)
            c, sn = ph.cos(), ph.sin()
            d0, d1 = h0 * c - h1 * sn - t0, h0 * sn + h1 * c - t1
            return m.cfg.gamma - (d0 * d0 + d1 * d1).sqrt().sum(-1)

        by = lambda x: x.view(bs // cs, cs, 1, -1)                                   # noqa: E731
        ng = neg.view(bs // cs, 1, ns, D)
        neg_score = torch.cat([score(by(h)[c:c + 1], by(r)[c:c + 1], ng[c:c + 1]) for c in range(bs // cs)])   # tails first
        ls = torch.nn.functional.logsigmoid
        loss = (-ls(score(h, r, t)).mean() - ls(-neg_score).mean()) / 2
        loss.backward()
    ent, ent_state = _adagrad(m.entity.weight, m.entity.state, torch.cat([s.h, s.t, s.neg]), torch.cat([h.grad, t.grad, neg.grad]),
                              m.cfg.lr, m.cfg.eps)
    rel, rel_state = _adagrad(m.relation.weight, m.relation.state, s.r, r.grad, m.cfg.lr, m.cfg.eps)
    return {"loss": loss.detach(), "entities": ent, "entity_state": ent_state, "relations": rel, "relation_state": rel_state}


_EXACT = {"dlrm": _exact_dlrm, "predict": _exact_dlrm, "mlp": _exact_mlp, "bag": _exact_bag, "interaction": _exact_interaction,
          "table": _exact_table, "ps": _exact_ps, "cache": _exact_cache, "kge": _exact_kge}
