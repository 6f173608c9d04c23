"""Performance cases of the framework: what its users run, through its public entry points.

Six families.  ``attention`` (the differentiable masked sparse attention, forward + backward or forward alone), ``spmm`` (graph
aggregation), ``ffn`` (two fused linear layers), ``residual`` (dropout-free residual + LayerNorm, with the attention
normalisation folded in), ``step`` (a whole training step of the distributed Exphormer on a 1 x 1 grid, captured once as a
program keeps it) and ``logits`` (inference of the node-level Graphormer on a sampled batch).

Graphs are Chung-Lu power-law graphs (exponent 2.1, ids without degree order), symmetrised, with expander edges and a global
token where the model has them; features are N(0, 1) and weights have the models' own initial scale.  Everything is made on
the GPU from the seed.  ``exact`` restates each family in 64 bits with plain torch.
"""
import math

import torch

DEV = "cuda"


# ---- the cases ------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the attention layer of the 169K-node Exphormer configuration (4 x 256 x 8 heads): graph + expander + token edges
        dict(name="attn_exphormer", kind="attention", nodes=169343, edges=1166243, expander=4, token=True, heads=8, dim=32, dtype="bf16",
             score="gated", norm="clampexp", train=True),
        # the same operator on a batch-sized sub-graph with the narrow model of the smoke test: launches and gaps count
        dict(name="attn_small", kind="attention", nodes=4097, edges=24570, expander=3, token=True, heads=4, dim=32, dtype="bf16",
             score="gated", norm="clampexp", train=True),
        # UniMP 3 x 128 x 4 on the co-purchase graph's density (23 edges a node), a quarter of its nodes: plain softmax attention
        dict(name="attn_unimp", kind="attention", nodes=612257, edges=6900000, expander=0, token=False, heads=4, dim=32, dtype="bf16",
             score="dot", norm="softmax", train=True),
        # Graphormer 6 x 512 x 16 with edge-type bias over a dense sampled mask: forward alone, as in evaluation
        dict(name="attn_graphormer_eval", kind="attention", nodes=150001, edges=3900000, expander=1, token=True, heads=16, dim=32,
             dtype="bf16", score="biased", norm="softmax", train=False),
        # fp32 operands (parity runs and small graphs), a head dim of 16 and an odd number of nodes
        dict(name="attn_fp32", kind="attention", nodes=40009, edges=300007, expander=2, token=False, heads=8, dim=16, dtype="fp32",
             score="gated", norm="clampexp", train=True),
        # GCN aggregation of the same Exphormer configuration, forward and backward
        dict(name="spmm_gcn", kind="spmm", nodes=169343, edges=1166243, width=256, dtype="bf16"),
        # feed-forward block 256 -> 512 -> 256 with ReLU over all nodes (ragged row count), forward and backward
        dict(name="ffn_256", kind="ffn", rows=169343, width=256, hidden=512, act="relu"),
        # feed-forward block 512 -> 1024 -> 512 with GELU on a batch of rows: the Graphormer block's dense half
        dict(name="ffn_512_batch", kind="ffn", rows=20011, width=512, hidden=1024, act="gelu"),
        # residual + LayerNorm after the attention: acc / l per head, + x, normalise; forward and backward
        dict(name="residual_norm", kind="residual", rows=169343, width=256, heads=8),
        # one training epoch (= step) of the 169K-node Exphormer configuration, dropout 0.1
        dict(name="step_exphormer", kind="step", nodes=169343, edges=1166243, expander=4, features=128, hidden=256, heads=8, layers=4,
             classes=40),
        # one training step on a small graph (the smoke test's model): launch gaps and small grids
        dict(name="step_small", kind="step", nodes=4096, edges=12288, expander=3, features=64, hidden=128, heads=4, layers=2, classes=16),
        # evaluation of the node-level Graphormer (hidden 64, 8 heads, 4 layers) on a 6,400-node batch: the smallest real call
        dict(name="logits_batch", kind="logits", nodes=6400, edges=21000, features=128, hidden=64, ffn=64, heads=8, layers=4, classes=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "spmm", "ffn", "residual", "step", "logits"])
    if kind == "attention":
        heads, dim = rng.choice([(8, 32), (8, 32), (4, 32), (16, 32), (8, 8), (8, 16), (4, 64), (2, 32), (2, 40)])
        score, norm = rng.choice([("gated", "clampexp"), ("gated", "clampexp"), ("dot", "softmax"), ("biased", "softmax"), ("dot", "clampexp")])
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp32"])
        nodes = _log(rng, 1500, 200000) if dtype == "bf16" else _log(rng, 1500, 60000)
        return dict(kind=kind, nodes=nodes, edges=int(nodes * rng.uniform(1.5, 12.0)), expander=rng.randint(1, 4), token=rng.random() < 0.5,
                    heads=heads, dim=dim, dtype=dtype, score=score, norm=norm, train=rng.random() < 0.75)
    if kind == "spmm":
        nodes = _log(rng, 2000, 300000)
        return dict(kind=kind, nodes=nodes, edges=int(nodes * rng.uniform(2.0, 10.0)), width=8 * _log(rng, 4, 64), dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "ffn":
        width = rng.choice([64, 128, 256, 512])
        return dict(kind=kind, rows=_log(rng, 1000, 170000), width=width, hidden=width * rng.choice([1, 2, 4]), act=rng.choice(["relu", "gelu"]))
    if kind == "residual":
        heads = rng.choice([4, 8, 16])
        return dict(kind=kind, rows=_log(rng, 1000, 250000), width=heads * rng.choice([8, 16, 32]), heads=heads)
    if kind == "step":
        nodes = _log(rng, 3000, 120000)
        heads = rng.choice([4, 8])
        return dict(kind=kind, nodes=nodes, edges=int(nodes * rng.uniform(3.0, 7.0)), expander=rng.randint(2, 4), features=8 * rng.randint(4, 16),
                    hidden=32 * heads, heads=heads, layers=rng.randint(2, 4), classes=rng.randint(5, 50))
    nodes = _log(rng, 2000, 64000)
    hidden, heads = rng.choice([(64, 8), (64, 8), (128, 8), (128, 4), (256, 8)])
    return dict(kind=kind, nodes=nodes, edges=int(nodes * rng.uniform(2.0, 7.0)), features=8 * rng.randint(8, 16), hidden=hidden,
                ffn=hidden * rng.choice([1, 2]), heads=heads, layers=rng.randint(2, 5), classes=rng.randint(5, 50))


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _randn(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def _dtype(case):
    return torch.float32 if case.get("dtype") == "fp32" else torch.bfloat16


def _power_law(g, n, m):
    """Symmetrised Chung-Lu edges without loops and duplicates, ids in random order: ``[2, about 2 m]`` (src, dst)."""
    i0 = max(1.0, n ** (1.0 - 1.0 / 1.1))
    w = (torch.arange(n, dtype=torch.float64, device=DEV) + i0).pow(-1.0 / 1.1)
    cdf = torch.cumsum(w, 0)
    u = torch.rand(2, m, dtype=torch.float64, generator=g, device=DEV) * cdf[-1]
    ei = torch.randperm(n, generator=g, device=DEV)[torch.searchsorted(cdf, u).clamp_(max=n - 1)]
    ei = ei[:, ei[0] != ei[1]]
    key = torch.unique(torch.cat([ei[0] * n + ei[1], ei[1] * n + ei[0]]))
    return torch.stack([key % n, key // n])


def _expander(g, n, deg):
    """``deg`` random edges per node in both directions."""
    src = torch.arange(n, device=DEV).repeat(deg)
    dst = torch.cat([torch.randperm(n, generator=g, device=DEV) for _ in range(deg)])
    return torch.cat([torch.stack([src, dst]), torch.stack([dst, src])], 1)


def _token(n):
    """Edges of a global token with id ``n`` to and from all nodes."""
    nodes = torch.arange(n, device=DEV)
    tok = torch.full_like(nodes, n)
    return torch.cat([torch.stack([nodes, tok]), torch.stack([tok, nodes])], 1)


def _mask(g, case):
    """``(edge_index, edge_type, number of nodes)`` of an attention mask: graph 0, expander 1, token 2."""
    n = case["nodes"]
    parts = [_power_law(g, n, case["edges"])]
    if case["expander"]:
        parts.append(_expander(g, n, case["expander"]))
    types = [torch.full((p.shape[1],), t, device=DEV) for t, p in enumerate(parts)]
    if case["token"]:
        parts.append(_token(n))
        types.append(torch.full((2 * n,), 2, device=DEV))
    return torch.cat(parts, 1), torch.cat(types), n + (1 if case["token"] else 0)


def _num_types(case):
    return 3 if case["token"] else (2 if case["expander"] else 1)


def _attention_inputs(case, seed):
    g = _gen(seed)
    ei, et, n = _mask(g, case)
    h, d, dt = case["heads"], case["dim"], _dtype(case)
    t = dict(ei=ei, et=et, n=n)
    for name in ("q", "k", "v", "do"):
        t[name] = _randn(g, n, h, d, dtype=dt)
    t["gate"] = _randn(g, _num_types(case), h, d) if case["score"] == "gated" else None
    t["bias"] = _randn(g, _num_types(case), h, scale=0.5) if case["score"] == "biased" else None
    return t


def _spmm_inputs(case, seed):
    g = _gen(seed)
    n = case["nodes"]
    loops = torch.arange(n, device=DEV)
    ei = torch.cat([_power_law(g, n, case["edges"]), torch.stack([loops, loops])], 1)
    deg = torch.bincount(ei[1], minlength=n).double()
    w = (deg[ei[0]] * deg[ei[1]]).rsqrt().float()
    return dict(n=n, ei=ei, w=w, x=_randn(g, n, case["width"], dtype=_dtype(case)), dout=_randn(g, n, case["width"], dtype=_dtype(case)))


def _ffn_inputs(case, seed):
    g = _gen(seed)
    m, d, h = case["rows"], case["width"], case["hidden"]
    return dict(x=_randn(g, m, d, dtype=torch.bfloat16), dy=_randn(g, m, d, dtype=torch.bfloat16), w1=_randn(g, h, d, scale=d ** -0.5),
                b1=_randn(g, h, scale=0.1), w2=_randn(g, d, h, scale=h ** -0.5), b2=_randn(g, d, scale=0.1))


def _residual_inputs(case, seed):
    g = _gen(seed)
    m, d, h = case["rows"], case["width"], case["heads"]
    return dict(acc=_randn(g, m, d, scale=8.0), l=torch.rand(m, h, generator=g, device=DEV) * 20 + 1, x=_randn(g, m, d, dtype=torch.bfloat16),
                dout=_randn(g, m, d, dtype=torch.bfloat16), gamma=1 + _randn(g, d, scale=0.1), beta=_randn(g, d, scale=0.1))


def _logits_inputs(case, seed):
    g = _gen(seed)
    n, f, h, ffn = case["nodes"], case["features"], case["hidden"], case["ffn"]
    sub = _power_law(g, n, case["edges"]) + 1                       # node 0 is the global token
    nodes = torch.arange(1, n + 1, device=DEV)
    zero = torch.zeros_like(nodes)
    ei = torch.cat([sub, torch.stack([nodes, zero]), torch.stack([zero, nodes])], 1)
    lin = lambda name, o, i: {name + ".weight": _randn(g, o, i, scale=i ** -0.5), name + ".bias": _randn(g, o, scale=0.1)}     # noqa: E731
    ln = lambda name, w: {name + ".weight": 1 + _randn(g, w, scale=0.1), name + ".bias": _randn(g, w, scale=0.1)}              # noqa: E731
    sd = {**lin("encoder", h, f), "graph_token.weight": _randn(g, 1, h)}
    for i in range(case["layers"]):
        p = f"layers.{i}."
        for name in ("q", "k", "v", "o"):
            sd.update(lin(p + name, h, h))
        sd.update({**ln(p + "ln1", h), **ln(p + "ln2", h), **lin(p + "ff1", ffn, h), **lin(p + "ff2", h, ffn)})
    sd.update({**ln("final_ln", h), **lin("out", case["classes"], h)})
    return dict(ei=ei, n=n + 1, x=_randn(g, n, f, dtype=torch.bfloat16), sd=sd)


# ---- states and passes -----------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"case": case, **_PREPARE[case["kind"]](case, seed)}


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


def _prepare_attention(case, seed):
    from gt_b200.attention import BlockCSR
    t = _attention_inputs(case, seed)
    blk = BlockCSR.from_edges(t["ei"], t["n"], t["n"], t["et"])
    leaves = {k: t[k].requires_grad_(case["train"]) for k in ("q", "k", "v", "gate", "bias") if t[k] is not None}
    return dict(blk=blk, do=t["do"], leaves=leaves)


def _run_attention(case, s):
    from gt_b200.attention.backend_cuda import masked_sparse_attention_cuda
    v = s["leaves"]
    o = masked_sparse_attention_cuda(v["q"], v["k"], v["v"], s["blk"], gate=v.get("gate"), bias=v.get("bias"), score=case["score"], norm=case["norm"])
    if not case["train"]:
        return o
    return [o.detach()] + list(torch.autograd.grad(o, list(v.values()), s["do"]))


def _prepare_spmm(case, seed):
    from gt_b200.attention import BlockCSR
    t = _spmm_inputs(case, seed)
    return dict(blk=BlockCSR.from_edges(t["ei"], t["n"], t["n"], weight=t["w"]), x=t["x"].requires_grad_(), dout=t["dout"])


def _run_spmm(case, s):
    from gt_b200.ops.sparse import spmm
    y = spmm(s["blk"], s["x"])
    return [y.detach(), torch.autograd.grad(y, s["x"], s["dout"])[0]]


def _prepare_ffn(case, seed):
    t = _ffn_inputs(case, seed)
    return dict(dy=t["dy"], leaves=[t[k].requires_grad_() for k in ("x", "w1", "b1", "w2", "b2")])


def _run_ffn(case, s):
    from gt_b200.ops import functional as K
    x, w1, b1, w2, b2 = s["leaves"]
    y = K.linear(K.linear(x, w1, b1, activation=case["act"]), w2, b2)
    return [y.detach()] + list(torch.autograd.grad(y, s["leaves"], s["dy"]))


def _prepare_residual(case, seed):
    from gt_b200.ops import functional as K
    t = _residual_inputs(case, seed)
    norm = K.LayerNorm(case["width"]).to(DEV)
    norm.load_state_dict(dict(weight=t["gamma"], bias=t["beta"]))
    return dict(norm=norm, dout=t["dout"], leaves=[t[k].requires_grad_() for k in ("acc", "x", "l")])


def _run_residual(case, s):
    from gt_b200.ops import functional as K
    acc, x, l = s["leaves"]
    y = K.dropout_add_norm(s["norm"], acc, x, l=l)
    return [y.detach()] + list(torch.autograd.grad(y, s["leaves"] + [s["norm"].weight, s["norm"].bias], s["dout"]))


def _prepare_step(case, seed):
    from gt_b200.models.exphormer_dist import DistExphormer, gcn_edges_with_self_loops
    from gt_b200.models.exphormer_ref import ExphormerRef
    from gt_b200.ops import native
    from gt_b200.parallel.grid import make_grid
    from gt_b200.parallel.layers import dist_cross_entropy
    from gt_b200.train.engine import TrainEngine, init_single_process_group
    init_single_process_group("nccl")
    g = _gen(seed)
    n = case["nodes"]
    base, exp, tok = _power_law(g, n, case["edges"]), _expander(g, n, case["expander"]), _token(n)
    n_tot = n + 1
    grid = make_grid((1, 1), n_tot, n_pad=-(-n_tot // 8) * 8).to(DEV)
    attn_ei, attn_et = ExphormerRef.build_attention_edges(base, exp, tok)
    rows = grid.n_pad
    torch.manual_seed(int(seed))
    model = DistExphormer(grid, gcn_edges_with_self_loops(base, n_tot), attn_ei, attn_et, case["features"], case["hidden"], case["classes"],
                          case["layers"], case["heads"], dropout=0.1, gnn_dropout=0.1, num_edge_types=3, backend="cuda", fused=True, norm="ln",
                          kernel_dtype=torch.bfloat16).to(DEV)
    x = torch.zeros(rows, case["features"], dtype=torch.bfloat16, device=DEV)
    x[:n] = _randn(g, n, case["features"], dtype=torch.bfloat16)
    y = torch.randint(0, case["classes"], (rows,), generator=g, device=DEV)
    mask = torch.rand(rows, generator=g, device=DEV) < 0.54
    mask[n:] = False
    n_train = int(mask.sum())
    # the step is captured once and replayed, as bench.py and the training command keep it; capturing takes three steps, after
    # which the weights and moments are put back to their initial values
    eng = TrainEngine(model, lr=1e-3, weight_decay=1e-3, total_steps=1 << 20, warmup=5, use_graph=True, graph_warmup=2)
    start, init = eng.state_dict(), eng.flat_p.clone()
    model.train()
    logits = {}

    def loss_fn():
        logits["out"] = model(x)
        return dist_cross_entropy(logits["out"], y, mask, n_train)

    for _ in range(3):
        eng.train_step(loss_fn)
    eng.flat_p.copy_(init)
    eng.load_state_dict(start)
    native.seed_rng(int(seed) + 1, DEV)
    return dict(eng=eng, model=model, loss_fn=loss_fn, logits=logits)



def _run_step(case, s):
    loss = s["eng"].train_step(s["loss_fn"])
    return dict(loss=loss, logits=s["logits"]["out"].detach(), grads=s["eng"].flat_g, weights=s["eng"].flat_p)


def _prepare_logits(case, seed):
    from gt_b200.models.graphormer_node import GraphormerNode
    t = _logits_inputs(case, seed)
    net = GraphormerNode(case["features"], case["hidden"], case["ffn"], case["heads"], case["layers"], case["classes"], t["ei"], t["n"]).to(DEV)
    net.load_state_dict(t["sd"])
    return dict(net=net.eval(), x=t["x"])


def _run_logits(case, s):
    with torch.no_grad():
        return s["net"](s["x"])


_PREPARE = dict(attention=_prepare_attention, spmm=_prepare_spmm, ffn=_prepare_ffn, residual=_prepare_residual, step=_prepare_step,
                logits=_prepare_logits)
_RUN = dict(attention=_run_attention, spmm=_run_spmm, ffn=_run_ffn, residual=_run_residual, step=_run_step, logits=_run_logits)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _edge_count(case):
    n = case["nodes"] + (1 if case.get("token") else 0)
    return 2 * case["edges"] + 2 * case["nodes"] * (case["expander"] + (1 if case.get("token") else 0)), n


def work(case):
    kind = case["kind"]
    b = 4 if case.get("dtype") == "fp32" else 2
    if kind == "attention":
        e, n = _edge_count(case)
        hd = case["heads"] * case["dim"]
        if not case["train"]:
            return dict(bytes=4 * n * hd * b + 8 * e, flops=4 * e * hd)         # q k v -> o; column and type of every edge
        return dict(bytes=8 * n * hd * b + 8 * e, flops=12 * e * hd)            # q k v do -> o dq dk dv
    if kind == "spmm":
        n, w = case["nodes"], case["width"]
        e = 2 * case["edges"] + n
        return dict(bytes=4 * n * w * b + 8 * e, flops=4 * e * w)
    if kind == "ffn":
        m, d, h = case["rows"], case["width"], case["hidden"]
        return dict(bytes=2 * 4 * m * d + 16 * d * h, flops=12 * m * d * h)     # x dy -> y dx; both weights and their gradients
    if kind == "residual":
        m, d = case["rows"], case["width"]
        return dict(bytes=m * (2 * 4 * d + 4 * 2 * d + 8 * case["heads"]), flops=30 * m * d)
    if kind == "step":
        n, d, layers = case["nodes"] + 1, case["hidden"], case["layers"]
        e_attn, e_gcn = 2 * case["edges"] + 2 * case["nodes"] * (case["expander"] + 1), 2 * case["edges"] + n
        gemm = 6 * n * d * (8 * d * layers + case["features"] + case["classes"])
        per_edge = layers * (12 * e_attn * d + 4 * e_gcn * d)
        # activations that have to be kept for the backward: read and written once per layer, structures once per layer
        return dict(bytes=layers * (16 * n * d * 2 + 8 * (e_attn + e_gcn)) + 2 * n * case["features"], flops=gemm + per_edge)
    n, h, f, layers = case["nodes"] + 1, case["hidden"], case["ffn"], case["layers"]
    e = 2 * case["edges"] + 2 * case["nodes"]
    weights = case["features"] * h + layers * (4 * h * h + 2 * h * f) + h * case["classes"]
    return dict(bytes=2 * n * (case["features"] + case["classes"]) + 4 * weights + 4 * e * layers, flops=2 * n * weights + 4 * e * h * layers)


def tolerance(case):
    """About four times what two correct implementations of the same precision differ by (bf16 storage of results and of the
    gradients in between: 2^-9 relative per rounding; fp32 sums: 1e-7 per rounding over some hundred terms)."""
    kind = case["kind"]
    if case.get("dtype") == "fp32":
        return {"rel": 2e-5, "max": 1e-2}
    if kind in ("step", "logits"):
        return {"rel": 2e-2, "max": 0.5}
    return {"rel": 1e-2, "max": 0.2}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
_CHUNK = 1 << 20        # edges at a time


def exact(case, seed):
    f = _EXACT.get(case["kind"])
    return f(case, seed) if f else None


def _attend64(q, k, v, ei, et, gate, bias, norm, do=None, clamp=(-5.0, 5.0), eps=1e-6):
    """``o`` (and the gradients for ``do``) of the masked attention, edges in chunks."""
    n, h, d = q.shape
    src, dst = ei
    scale = d ** -0.5
    new = lambda *s: torch.zeros(*s, dtype=torch.float64, device=q.device)      # noqa: E731
    spans = [slice(i, i + _CHUNK) for i in range(0, src.numel(), _CHUNK)]
    s_all = new(src.numel(), h)
    for c in spans:
        kg = k[src[c]] * gate[et[c]] if gate is not None else k[src[c]]
        s_all[c] = (q[dst[c]] * kg).sum(-1) * scale
        if bias is not None:
            s_all[c] += bias[et[c]]
    if norm == "softmax":
        m = torch.full((n, h), -math.inf, dtype=torch.float64, device=q.device)
        m.scatter_reduce_(0, dst[:, None].expand(-1, h), s_all, "amax")
        w, live, eps = torch.exp(s_all - m[dst]), None, 0.0
    else:
        w, live = torch.exp(s_all.clamp(*clamp)), (s_all >= clamp[0]) & (s_all <= clamp[1])
    den = new(n, h).index_add_(0, dst, w) + eps
    w /= torch.where(den > 0, den, torch.ones_like(den))[dst]
    o = new(n, h, d)
    for c in spans:
        o.index_add_(0, dst[c], w[c].unsqueeze(-1) * v[src[c]])
    if do is None:
        return o
    delta = (do * o).sum(-1)
    dq, dk, dv = new(n, h, d), new(n, h, d), new(n, h, d)
    dgate = new(*gate.shape) if gate is not None else None
    dbias = new(*bias.shape) if bias is not None else None
    for c in spans:
        dov, p = do[dst[c]], w[c]
        ds = p * ((dov * v[src[c]]).sum(-1) - delta[dst[c]])
        if live is not None:
            ds = ds * live[c]
        dv.index_add_(0, src[c], p.unsqueeze(-1) * dov)
        if dbias is not None:
            dbias.index_add_(0, et[c], ds)
        ds = ds.unsqueeze(-1) * scale
        qd, ks = q[dst[c]], k[src[c]]
        if gate is not None:
            gt = gate[et[c]]
            qk = ds * qd * ks
            for t in range(gate.shape[0]):
                dgate[t] += (qk * (et[c] == t)[:, None, None]).sum(0)
            qd, ks = qd * gt, ks * gt
        dq.index_add_(0, dst[c], ds * ks)
        dk.index_add_(0, src[c], ds * qd)
    return [o, dq, dk, dv] + [t for t in (dgate, dbias) if t is not None]


def _exact_attention(case, seed):
    t = _attention_inputs(case, seed)
    f = lambda x: x.double() if x is not None else None                          # noqa: E731
    return _attend64(f(t["q"]), f(t["k"]), f(t["v"]), t["ei"], t["et"], f(t["gate"]), f(t["bias"]), case["norm"],
                     f(t["do"]) if case["train"] else None)


def _exact_spmm(case, seed):
    t = _spmm_inputs(case, seed)
    (src, dst), w = t["ei"], t["w"].double()
    x, dout = t["x"].double(), t["dout"].double()
    y, dx = torch.zeros_like(x), torch.zeros_like(x)
    for i in range(0, src.numel(), _CHUNK):
        c = slice(i, i + _CHUNK)
        y.index_add_(0, dst[c], x[src[c]] * w[c, None])
        dx.index_add_(0, src[c], dout[dst[c]] * w[c, None])
    return [y, dx]


def _exact_ffn(case, seed):
    t = _ffn_inputs(case, seed)
    v = [t[k].double().requires_grad_() for k in ("x", "w1", "b1", "w2", "b2")]
    x, w1, b1, w2, b2 = v
    hid = x @ w1.t() + b1
    hid = torch.relu(hid) if case["act"] == "relu" else torch.nn.functional.gelu(hid)
    y = hid @ w2.t() + b2
    return [y.detach()] + list(torch.autograd.grad(y, v, t["dy"].double()))


def _exact_residual(case, seed):
    t = _residual_inputs(case, seed)
    v = [t[k].double().requires_grad_() for k in ("acc", "x", "l", "gamma", "beta")]
    acc, x, l, gamma, beta = v
    a = (acc.view(acc.shape[0], l.shape[1], -1) / (l + 1e-6).unsqueeze(-1)).reshape(acc.shape)
    y = torch.nn.functional.layer_norm(x + a, (case["width"],), gamma, beta, 1e-5)
    return [y.detach()] + list(torch.autograd.grad(y, v, t["dout"].double()))


def _exact_logits(case, seed):
    t = _logits_inputs(case, seed)
    sd = {k: v.double() for k, v in t["sd"].items()}
    lin = lambda x, name: x @ sd[name + ".weight"].t() + sd[name + ".bias"]       # noqa: E731
    ln = lambda x, name: torch.nn.functional.layer_norm(x, (x.shape[1],), sd[name + ".weight"], sd[name + ".bias"], 1e-5)     # noqa: E731
    h = torch.cat([sd["graph_token.weight"], lin(t["x"].double(), "encoder")])
    heads = lambda x: x.view(x.shape[0], case["heads"], -1)                        # noqa: E731
    for i in range(case["layers"]):
        p = f"layers.{i}."
        y = ln(h, p + "ln1")
        o = _attend64(heads(lin(y, p + "q")), heads(lin(y, p + "k")), heads(lin(y, p + "v")), t["ei"], None, None, None, "clampexp")
        h = h + lin(o.reshape(h.shape), p + "o")
        h = h + lin(torch.nn.functional.gelu(lin(ln(h, p + "ln2"), p + "ff1")), p + "ff2")
    return lin(ln(h, "final_ln")[1:], "out")


_EXACT = dict(attention=_exact_attention, spmm=_exact_spmm, ffn=_exact_ffn, residual=_exact_residual, logits=_exact_logits)
