"""Edge attention as streams of segments, at the sizes where the split ends: one row, partial warps, heads that do not fill a
lane group, several segments per lane group, empty rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(n, max_deg, seed, typed):
    from budgetformer_b200.graph.attn_graph import AttnGraph
    gen = torch.Generator().manual_seed(seed)
    deg = torch.randint(0, max_deg + 1, (n,), generator=gen)
    dst = torch.repeat_interleave(torch.arange(n), deg)
    src = (torch.rand(dst.numel(), generator=gen) ** 3 * n).long().clamp_(max=n - 1)     # popular keys: split work items
    rows = [src, dst] + ([torch.randint(0, 2, (dst.numel(),), generator=gen)] if typed else [])
    return AttnGraph.from_edge_index(torch.stack(rows), n).to("cuda")


def _reference(q, k, v, dout, graph, tab, variant, p, seed):
    from budgetformer_b200.ops.edge_attention import edge_attention_reference
    t = [x.detach().double().requires_grad_() for x in (q, k, v)]
    # the reference computes in fp32: exact enough beside 16-bit results, and 1e-5 of fp32 ones
    tt = None if tab is None else tab.detach().clone().requires_grad_()
    out = edge_attention_reference(*t, graph, variant=variant, etable=tt, dropout_p=p, dropout_seed=seed)
    grads = torch.autograd.grad(out, t + ([tt] if tt is not None else []), dout.double())
    return [out] + list(grads)


@pytest.mark.parametrize("variant", ["plain", "gps", "exphormer"])
@pytest.mark.parametrize("n,heads,hn,max_deg,dtype", [
    (1, 1, 8, 3, torch.bfloat16), (5, 3, 16, 0, torch.bfloat16), (33, 5, 32, 9, torch.float16), (257, 8, 16, 40, torch.bfloat16),
    (1031, 1, 8, 130, torch.float32), (700, 3, 64, 12, torch.float32), (300, 2, 128, 7, torch.bfloat16), (100, 12, 64, 5, torch.float32),
    (30011, 8, 32, 8, torch.bfloat16), (30011, 8, 8, 6, torch.float16), (9001, 4, 64, 8, torch.float32)])
def test_attention_streams(n, heads, hn, max_deg, dtype, variant):
    from budgetformer_b200.ops.edge_attention import edge_attention
    if variant == "exphormer" and max_deg == 0:
        max_deg = 1                                                        # typed edges cannot be an empty list
    graph = _graph(n, max_deg, 7 * n + heads, variant == "exphormer")
    gen = torch.Generator(device="cuda").manual_seed(n + hn)
    q, k, v, dout = (torch.randn(n, heads, hn, generator=gen, device="cuda").to(dtype) for _ in range(4))
    tab = torch.randn(2, heads, hn, generator=gen, device="cuda") if variant == "exphormer" else None
    p = 0.3 if variant == "gps" else 0.0
    want = _reference(q, k, v, dout, graph, tab, variant, p, 11)
    args = [x.requires_grad_() for x in (q, k, v)] + ([tab.requires_grad_()] if tab is not None else [])
    out = edge_attention(q, k, v, graph, variant=variant, etable=tab, dropout_p=p, dropout_seed=11)
    got = [out] + list(torch.autograd.grad(out, args, dout))
    # 16 bits: the context is rounded when stored (unit 2^-9 / 2^-12) and D = <dout, out> inherits it; fp32: sums of <= 10^3 terms.
    # A score within rounding of the clamp's edge loses its gradient on one side only, hence norms and not single entries.
    # Score gradients are differences <dout, v_j> - D that cancel (to zero in a row of one edge): what the rounding of D leaves is
    # at most unit * |dout_i| |out_i| |k_j| / sqrt(hn) a row, of the order of unit * |dout| in all: the second term.
    tol = {torch.float32: 2e-5, torch.float16: 4e-3, torch.bfloat16: 2.5e-2}[dtype]
    for a, b in zip(got, want):
        scale = float(b.double().norm()) + float(dout.double().norm())
        assert float((a.double() - b.double()).norm()) <= tol * scale + 1e-6, (float((a.double() - b.double()).norm()), scale)


def test_attention_streams_keep_other_rows_finite():
    """An infinite key / value row reaches the queries that name it and nobody else: stale ring slots are never added."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    n = 203
    dst = torch.arange(n).repeat_interleave(torch.arange(n) % 7)
    src = (torch.arange(dst.numel()) * 5 + 1) % n
    src[src == 9] = 10
    src[dst == 50] = 9                                                     # only query 50 names key 9
    graph = AttnGraph.from_edge_index(torch.stack([src, dst]), n).to("cuda")
    q, k, v = (torch.randn(n, 4, 16, device="cuda").bfloat16() for _ in range(3))
    k[9], v[9] = float("nan"), float("inf")
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    out = edge_attention(q, k, v, graph)
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), torch.ones_like(out))
    others = torch.arange(n, device="cuda") != 50
    assert torch.isfinite(out[others]).all() and torch.isfinite(dq[others]).all()
    keys = torch.ones(n, dtype=torch.bool, device="cuda")
    keys[9] = False
    assert torch.isfinite(dk[keys]).all() and torch.isfinite(dv[keys]).all()
