"""Row kernels at the edges of their tilings, against 64-bit PyTorch restatements (single GPU).

Tolerances: a result that is a sum of n fp32 products of either sign has a relative error (2-norm) of a few units of 2^-24
times sqrt(n) at most; 2e-6 holds for the up to 4,000 terms met here.  bf16 results carry one rounding, 2^-9 relative per
element, 2^-8.5 allowed in the norm.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

F32, BF16 = 2e-6, 2.0 ** -8.5


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-300)).item()


def _adagrad(w, st, rows, g, norm, lr, eps):
    w, st = w.double(), st.double()
    st.index_add_(0, rows, norm)
    return w.index_add_(0, rows, -lr * g / (st[rows].sqrt() + eps).unsqueeze(1)), st


@pytest.mark.parametrize("D,T,B,hot,shift,weighted", [
    (4, 1, 1, [1], 0, False),                      # smallest row, one bag
    (16, 3, 45, [1, 0, 3], 0, False),              # a table without ids
    (32, 2, 1000, None, 0, True),                  # jagged, weighted, empty bags
    (64, 40, 33, [1, 2] * 20, 0, False),           # more than 32 tables: two steps of the table search
    (100, 5, 77, None, 0, False),                  # rows of 25 sixteen-byte units
    (120, 3, 129, [1, 1, 9], 4, False),            # rows of 15 units; places and gradients off the 16-byte boundary
    (128, 2, 3000, [1, 70], 4, False),             # one-id table beside long bags
    (256, 3, 50, None, 0, True),
    (300, 2, 40, [2, 1], 0, False),                # two sixteen-byte units per lane and a tail
    (512, 1, 65, [33], 0, False),                  # widest row, bags longer than a warp
])
@pytest.mark.parametrize("bf16", [False, True])
def test_pooled_lookup_and_update(D, T, B, hot, shift, weighted, bf16):
    from recstore_b200.ops import functional as F_
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(D + T)
    i64, i32 = dict(dtype=torch.int64, device=dev), dict(dtype=torch.int32, device=dev)
    rows = [(7 + 37 * t) % 500 + 3 for t in range(T)]
    base = torch.tensor([sum(rows[:t]) for t in range(T)], **i64)
    weight = torch.randn(sum(rows), D, device=dev, generator=g)
    if hot is None:
        lens = torch.randint(0, 70, (T * B,), device=dev, generator=g) * (torch.rand(T * B, device=dev, generator=g) < 0.4)
    else:
        lens = torch.tensor(hot, **i64).repeat_interleave(B)
    offsets = torch.cat([torch.zeros(1, **i64), lens.cumsum(0)])
    nnz = int(offsets[-1])
    bag = torch.repeat_interleave(torch.arange(T * B, device=dev), lens)
    table = bag // B
    ids = (torch.rand(nnz, device=dev, generator=g) ** 3 * torch.tensor(rows, device=dev)[table]).long()
    psw = torch.rand(nnz, device=dev, generator=g) + 0.5 if weighted else None
    stride = T * D + shift
    out = torch.full((B, stride), 7.0, device=dev, dtype=torch.bfloat16 if bf16 else torch.float32)
    col = torch.arange(T, **i32) * D + shift
    ri, ob, st = torch.empty(nnz + 1, **i64), torch.empty(nnz + 1, **i32), torch.zeros(1, **i64)
    layout = dict(offsets=offsets) if hot is None else dict(hotness=torch.tensor(hot, **i32), hot_base=offsets[::B][:T].contiguous())
    F_.emb_forward(weight, base, torch.tensor(rows, **i64), ids, **layout, per_sample_weights=psw, T=T, B=B, D=D, B_local=B,
                   dst_table=torch.tensor([out.data_ptr()], **i64), dst_row_stride=stride, dst_col=col, out_bf16=bf16, row_idx=ri,
                   occ2bag=ob, status=st)
    w64 = psw.double() if weighted else torch.ones(nnz, dtype=torch.float64, device=dev)
    at = ids + base[table]
    assert torch.equal(ri[:nnz], at) and torch.equal(ob[:nnz].long(), bag)
    ref = torch.zeros(T * B, D, dtype=torch.float64, device=dev).index_add_(0, bag, weight[at].double() * w64.unsqueeze(1))
    got = out[:, shift:].reshape(B, T, D).transpose(0, 1).reshape(T * B, D)
    assert _rel(got, ref) < (BF16 if bf16 else F32)
    assert torch.all(got[lens == 0] == 0) and torch.all(out[:, :shift] == 7.0)

    grad = torch.randn(B, stride, device=dev, generator=g).to(out.dtype)
    per_bag = grad[:, shift:].reshape(B, T, D).transpose(0, 1).reshape(T * B, D).double()
    gnorm = per_bag.pow(2).sum(1).view(T, B).t().float().contiguous()
    for opt, norms in (("sgd", None), ("rowwise_adagrad", None), ("rowwise_adagrad", gnorm)):
        w, s = weight.clone(), torch.rand(weight.shape[0], device=dev, generator=g)
        s0 = s.clone()
        F_.emb_backward(w, s if opt != "sgd" else None, ri, ob, nnz, grad, grad_col=col, grad_row_stride=stride, B=B, D=D, grad_bf16=bf16,
                        per_sample_weights=psw, lr=0.5, eps=1e-8, optimizer=opt, status=st, gnorm=norms, gnorm_stride=T)
        gr = per_bag[bag] * w64.unsqueeze(1)
        if opt == "sgd":
            assert _rel(w, weight.double().index_add_(0, at, -0.5 * gr)) < F32
        else:
            rw, rs = _adagrad(weight, s0, at, gr, gr.pow(2).mean(1), 0.5, 1e-8)
            assert _rel(s, rs) < F32 and _rel(w, rw) < F32
    assert st.item() == 0


@pytest.mark.parametrize("n", [1, 31, 1000, 80000])
@pytest.mark.parametrize("D", [4, 32, 100, 400, 520])
@pytest.mark.parametrize("hashed", [False, True])
def test_one_rank_shard_verbs(n, D, hashed):
    """lookup / update / get / put / push_update on one rank against a host model, with duplicate, negative and absent keys."""
    from recstore_b200 import _lib
    from recstore_b200.parallel.peer import PeerContext
    from recstore_b200.parallel.sharded_table import ShardedEmbeddingTable
    if n * D > 8e6 * (1 + (D == 100)):
        n = 20000
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(n + D)
    N = 5000
    ctx = PeerContext(0, 1)
    t = ShardedEmbeddingTable(ctx, "t", N, D, max_keys=max(n, N), lr=0.1, eps=1e-8, hashed=hashed, init="zeros")
    model = torch.randn(N, D, device=dev, generator=g)
    key = (lambda i: i * 7919 + 3) if hashed else (lambda i: i)
    everything = torch.arange(N, device=dev)
    t.put(key(everything), model)
    ids = (torch.rand(n, device=dev, generator=g) ** 4 * N).long()
    pad = torch.rand(n, device=dev, generator=g) < 0.05
    keys = torch.where(pad, torch.full_like(ids, -5), key(ids))
    rows = t.lookup(keys)
    assert torch.equal(rows, model[ids] * (~pad).unsqueeze(1))
    if D <= 512:
        grad = torch.randn(n, D, device=dev, generator=g)
        keys_before = keys.clone()
        keys.fill_(0)                                       # the table keeps its own copy of what it looked up
        t.update(grad)
        live = ids[~pad]
        w, s = _adagrad(model, torch.zeros(N, device=dev), live, grad[~pad].double(), grad[~pad].double().pow(2).mean(1), 0.1, 1e-8)
        got, found = t.get(key(everything))
        assert bool(found.all()) and _rel(got, w) < F32
        t.push_update(keys_before, grad)
        w, s = _adagrad(w.float(), s.float(), live, grad[~pad].double(), grad[~pad].double().pow(2).mean(1), 0.1, 1e-8)
        got, _ = t.get(key(everything))
        assert _rel(got, w) < F32
        t.put(key(everything[:7]), model[:7])               # a put row's optimizer state starts over
        got, _ = t.get(key(everything[:7]))
        assert torch.equal(got, model[:7])
    ctx.check_status()
    if hashed:
        absent = torch.tensor([10 ** 12, key(3), 10 ** 12 + 1], device=dev)
        r, found = t.get(absent)
        assert found.tolist() == [False, True, False] and float(r[0].abs().sum()) == 0.0
        twice = torch.tensor([10 ** 12] * 64, device=dev)   # first touch, many times in one call: one key, one value
        a = t.lookup(twice)
        assert torch.equal(a, a[:1].expand_as(a)) and float(a.abs().sum()) > 0 and bool((a.abs() <= t.init_scale).all())
        assert torch.equal(t.get(twice[:1])[0], a[:1])
        ctx.check_status()
    else:
        assert float(t.lookup(torch.tensor([N, 0], device=dev))[0].abs().sum()) == 0.0
        with pytest.raises(_lib.DeviceStatusError):
            ctx.check_status()
    t.lookup(torch.tensor([-1], device=dev))                # a reserved key is refused
    with pytest.raises(_lib.DeviceStatusError):
        ctx.check_status()
    ctx.free_all()


@pytest.mark.parametrize("M,K", [(1, 8), (37, 256), (5000, 264), (999, 512), (300, 1024), (70001, 256)])
def test_head_sizes(M, K):
    from recstore_b200.ops import functional as F_
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(K)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    w, b = torch.randn(K, device=dev, generator=g) * 0.1, torch.randn(1, device=dev, generator=g)
    y = (torch.rand(M, device=dev, generator=g) < 0.25).float()
    prob, ls, dw, db = torch.empty(M, device=dev), torch.zeros(1, device=dev), torch.zeros(K, device=dev), torch.zeros(1, device=dev)
    dx = torch.empty(M, K, device=dev, dtype=torch.bfloat16)
    F_.head_bce(x, w, b, y, 1.0 / M, prob=prob, loss_sum=ls, dx=dx, dw=dw, db=db)
    x64 = x.double()
    z = x64 @ w.double() + b.double()
    dz = (torch.sigmoid(z) - y) / M
    # __expf in the logistic function: 2 ulp of its argument's size, so 1e-6 relative at the logits met here
    assert _rel(prob, torch.sigmoid(z)) < 1e-5
    assert _rel(ls, torch.nn.functional.binary_cross_entropy_with_logits(z, y.double()).view(1)) < 1e-5
    assert _rel(dw, x64.t() @ dz) < 1e-4 and _rel(db, dz.sum().view(1)) < 1e-4          # p - y: cancellation times 1e-5
    assert _rel(dx, dz.unsqueeze(1) * w.double() * (x64 > 0)) < BF16
    only = torch.empty(M, device=dev)
    F_.head_bce(x, w, b, None, 1.0 / M, prob=only)
    assert torch.equal(only, prob)
    src = torch.randn(M, 13, device=dev, generator=g)
    for ld in (16, 64, 20):
        out = torch.full((M, ld), 3.0, device=dev, dtype=torch.bfloat16)
        F_.pad_cast_bf16(src, out)
        assert torch.equal(out[:, :13], src.bfloat16()) and float(out[:, 13:].abs().sum()) == 0.0


@pytest.mark.parametrize("F,D,B,rows", [(2, 16, 1, 0), (32, 128, 19, 0), (27, 128, 2000, 0), (27, 128, 301, 2), (9, 48, 500, 1), (31, 112, 7, 0)])
def test_interaction_backward_edges(F, D, B, rows):
    """Several samples per warp, partial column blocks, a NaN and an infinity that must stay in their own sample."""
    from recstore_b200.ops import functional as F_
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(F)
    T = torch.randn(B, F, D, device=dev, generator=g).bfloat16()
    ld = (D + F * (F - 1) // 2 + 7) // 8 * 8
    dout = torch.randn(B, ld, device=dev, generator=g).bfloat16()
    if B > 1:
        T[0, 1, 0], T[0, 0, 1] = float("nan"), float("inf")
    dx = torch.zeros(B, D, device=dev, dtype=torch.bfloat16)
    G = torch.zeros(B, (F - 1) * D, device=dev, dtype=torch.bfloat16)
    nrm = torch.zeros(B, F - 1, device=dev)
    i32 = dict(dtype=torch.int32, device=dev)
    F_.interaction_backward(T, dout, B, F, D, dx, torch.tensor([G.data_ptr()], device=dev), torch.zeros(F - 1, **i32),
                            torch.arange(F - 1, **i32) * D, (F - 1) * D, 0, True, torch.tensor([nrm.data_ptr()], device=dev), F - 1, rows)
    t = T.double()
    li, lj = torch.tril_indices(F, F, offset=-1, device=dev)
    dz = torch.zeros(B, F, F, dtype=torch.float64, device=dev)
    dz[:, li, lj] = dout[:, D:D + li.numel()].double()
    dt = torch.bmm(dz + dz.transpose(1, 2), t)
    ref = (dt[:, 0] + dout[:, :D].double()) * (t[:, 0] > 0)
    s = 1 if B > 1 else 0
    if rows != 2:
        assert _rel(dx[s:], ref[s:]) < BF16
    if rows != 1:
        assert _rel(G.view(B, F - 1, D)[s:], dt[s:, 1:]) < BF16
        assert _rel(nrm[s:], dt[s:, 1:].pow(2).sum(-1)) < 2 * BF16
    else:
        assert float(G.abs().sum()) == 0.0


@pytest.mark.parametrize("model", ["TransE_l2", "DistMult", "SimplE", "TransE_l1", "RotatE"])
@pytest.mark.parametrize("bs,cs,ns,D", [(8, 8, 8, 8), (80, 40, 8, 44), (24, 24, 264, 136), (16, 16, 24, 520)])
def test_kge_scores_and_gradients_at_odd_sizes(model, bs, cs, ns, D):
    from recstore_b200.baseline.kge_torch import chunk_neg_score, edge_score, logsigmoid_loss
    from recstore_b200.models.kge import KGEConfig, KGEModel
    pair = model in ("TransE_l1", "RotatE")
    if not pair:
        ns = cs                                             # the gradient GEMM wants as many negatives as positives per chunk
    if D > 512 or (model == "RotatE" and D % 8) or (pair and cs % 8):
        D, cs, bs = min(D, 512) // 8 * 8, (cs + 7) // 8 * 8, (cs + 7) // 8 * 8 * (bs // cs)
    dev = torch.device("cuda:0")
    m = KGEModel(KGEConfig(n_entities=500, n_relations=20, dim=D, model=model, batch=bs, neg_sample_size=ns, neg_chunk_size=cs, seed=2))
    g = torch.Generator(device=dev).manual_seed(bs)
    pick = lambda n, hi: torch.randint(0, hi, (n,), device=dev, generator=g)             # noqa: E731
    hi, ti, ri, ni = pick(bs, 500), pick(bs, 500), pick(bs, 20), pick(bs // cs * ns, 500)
    for ch in (False, True):
        E, R = m.entity.weight, m.relation.weight
        h, t, n, r = (x.double().requires_grad_(True) for x in (E[hi], E[ti], E[ni], R[ri]))
        pos = edge_score(model, h, r, t, 10.0, None, m.emb_init)
        neg = chunk_neg_score(model, h, r, t, n, ch, cs, 10.0, None, m.emb_init)
        ref = logsigmoid_loss(pos, neg)
        ref.backward()
        p, q = m.score_batch(hi, ri, ti, ni, ch)
        tol = 1e-5 if pair else 2.0 ** -6                   # fp32 pairs; bf16 operands of the cross products
        assert _rel(p, pos.detach()) < 1e-5 and _rel(q, neg.detach().view_as(q)) < tol
        loss = m.train_step(hi, ri, ti, ni, ch)
        assert abs(loss.item() - ref.item()) < tol * max(1.0, abs(ref.item()))
        assert _rel(m.ent_grad, torch.cat([h.grad, t.grad, n.grad])) < (1e-4 if pair else 2.0 ** -6)
        assert _rel(m.rel_grad, r.grad) < (1e-4 if pair else 2.0 ** -6)
    m.ctx.check_status()
    m.ctx.free_all()


def test_replayed_inference_follows_the_parameters():
    """The first call runs eagerly, later ones replay a graph: same probabilities, for new inputs and after training steps."""
    from recstore_b200.models.dlrm import DLRM, DLRMConfig
    from recstore_b200.utils.data import DLRMBatchSource
    rows = [100, 7, 3000]
    engines = [DLRM(DLRMConfig(table_rows=rows, batch=100, seed=4, use_cuda_graph=graph)) for graph in (False, True)]
    src = DLRMBatchSource(rows, [1] * 3, 100, seed=5)
    for step in range(4):
        b = src.next()
        probs = [e.predict(e.make_pinned_batch(b.dense, b.ids, b.labels)) for e in engines]
        # the weight gradients' atomics may round differently in the two engines once they have trained
        assert torch.equal(*probs) if step < 2 else torch.allclose(*probs, atol=1e-3)
        if step > 0:
            for e in engines:
                e.train_step(e.make_pinned_batch(b.dense, b.ids, b.labels))
    for e in engines:
        e.check()
        e.ctx.free_all()


@pytest.mark.parametrize("model", ["TransE_l2", "RotatE", "RESCAL"])
def test_captured_kg_step_with_two_branches_matches_the_eager_one(model):
    from recstore_b200.models.kge import KGEConfig, KGEModel
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(9)
    pick = lambda n, hi: torch.randint(0, hi, (n,), device=dev, generator=g)             # noqa: E731
    pair = [KGEModel(KGEConfig(n_entities=300, n_relations=9, dim=64, model=model, batch=64, neg_sample_size=32, neg_chunk_size=32,
                               seed=3, use_cuda_graph=graph)) for graph in (False, True)]
    for step in range(5):
        ids = (pick(64, 300), pick(64, 9), pick(64, 300), pick(64, 300))
        losses = [m.train_step(*ids) for m in pair]
        assert abs(losses[0].item() - losses[1].item()) < 1e-4 * abs(losses[0].item())    # sums in another order, five steps
    assert _rel(pair[1].entity.weight, pair[0].entity.weight.double()) < 1e-3
    assert _rel(pair[1].relation.weight, pair[0].relation.weight.double()) < 1e-3
    # ids of another type take the copies
    pair[1].train_step(*[x.int() for x in ids])
    for m in pair:
        m.ctx.check_status()
        m.ctx.free_all()
