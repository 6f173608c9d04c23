"""Edge-gather attention kernels at the sizes where their loops change: segment lengths around the group (4 edges a lane group), the
chunk (32 edges) and the segment limit, empty rows, every lane layout, type changes at every position (run on a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(n, types, seed):
    """Row ``i`` has ``i % 71`` edges (0 .. 70), row 5 is a hub with an edge from every node; types in input order are mixed."""
    g = torch.Generator().manual_seed(seed)
    deg = torch.arange(n) % 71
    dst = torch.cat([torch.repeat_interleave(torch.arange(n), deg), torch.full((n,), 5)])
    src = torch.cat([torch.randint(0, n, (int(deg.sum()),), generator=g), torch.arange(n)])
    return torch.stack([src, dst]), torch.randint(0, types, (dst.numel(),), generator=g)


@pytest.mark.parametrize("h,d", [(8, 32), (4, 32), (16, 32), (1, 32), (32, 8), (4, 8), (8, 16), (4, 64), (8, 64), (2, 128), (1, 256)])
@pytest.mark.parametrize("score,norm,types", [("gated", "clampexp", 3), ("biased", "softmax", 4), ("dot", "softmax", 1)])
def test_passes_match_the_oracle(h, d, score, norm, types):
    from gt_b200.attention import BlockCSR
    from gt_b200.attention import backend_cuda as bc, backend_torch as bt
    dev = torch.device("cuda:0")
    n = 500
    ei, et = _graph(n, types, seed=h * 100 + d)
    blk = BlockCSR.from_edges(ei, n, n, et).to(dev)
    g = torch.Generator(device=dev).manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev)                       # noqa: E731
    q, k, v = (rnd(n, h, d).bfloat16() for _ in range(3))
    gate = rnd(types, h, d) if score == "gated" else None
    bias = rnd(types, h) if score == "biased" else None
    kw = dict(score=score, norm=norm)
    f = lambda t: t.double() if t is not None else None                              # noqa: E731
    ref = bt.attn_fwd_partial(f(q), f(k), f(v), blk, f(gate), f(bias), **kw)
    acc, l, m = bc.attn_fwd_partial(q, k, v, blk, gate, bias, **kw)
    # fp32 sums of at most 570 terms of exact bf16 operands: relative error below 570 * 2^-24 = 3.4e-5 of the largest row sum, plus
    # 2^-21 of the argument per exponential (arguments up to 5, or differences to the maximum)
    for got, want, name in zip((acc, l, m), ref, ("acc", "l", "m")):
        assert (got.double() - want).abs().max() <= 1e-4 * want.abs().max().clamp_min(1e-3), name
    dacc, dl = rnd(n, h, d), rnd(n, h)
    got = bc.attn_bwd_partial(q, k, v, blk, gate, bias, m, dacc, dl, **kw)
    want = bt.attn_bwd_partial(f(q), f(k), f(v), blk, f(gate), f(bias), ref[2], f(dacc.bfloat16()), f(dl), **kw)
    # dq / dk / dv are stored as bf16 (2^-9 relative per element); the table gradients are fp32 sums over all edges, whose terms
    # cancel: bounded by the same 1e-4 of the sum of magnitudes, taken as 20 times the largest result
    for a, b, name in zip(got, want, ("dq", "dk", "dv", "dgate", "dbias")):
        if b is not None:
            assert (a.double() - b).abs().max() <= 2.0 ** -8 * b.abs().max(), name


@pytest.mark.parametrize("h,d", [(8, 32), (4, 32), (2, 16)])
def test_infinite_values_stay_in_their_rows(h, d):
    """An infinite V row reaches exactly the rows that have an edge to it, also where the last group of a row is padded."""
    from gt_b200.attention import BlockCSR
    from gt_b200.attention import backend_cuda as bc
    dev = torch.device("cuda:0")
    n = 300
    ei, et = _graph(n, 1, seed=3)
    blk = BlockCSR.from_edges(ei, n, n, et).to(dev)
    q, k = torch.randn(n, h, d, device=dev).bfloat16(), torch.randn(n, h, d, device=dev).bfloat16()
    v = torch.ones(n, h, d, device=dev).bfloat16()
    v[17] = float("inf")
    acc, _, _ = bc.attn_fwd_partial(q, k, v, blk, score="dot", norm="clampexp")
    hit = torch.zeros(n, dtype=torch.bool)
    hit[ei[1][ei[0] == 17]] = True
    assert torch.isinf(acc[hit.to(dev)]).all() and torch.isfinite(acc[~hit.to(dev)]).all()
