"""sm_100a kernels against plain PyTorch fp32 references of the same ops."""
import pytest
import torch

from budgetformer_b200.graph.attn_graph import Topology
from budgetformer_b200.graph.builder import build_attn_graph
from budgetformer_b200.ops.edge_attention import edge_attention, edge_attention_reference
from tests.helpers import random_attn_graph, random_topology

pytestmark = pytest.mark.gpu

TOL = {torch.float32: (2e-4, 2e-4), torch.bfloat16: (3e-2, 3e-2), torch.float16: (5e-3, 5e-3)}


def _run(variant, dtype, hl, hn, hub_row=0, hub_col=0, dropout=0.0, n=257, e=2100):
    dev = torch.device("cuda")
    g = random_attn_graph(n, e, hub_row, hub_col, seed=hl * 7 + hn, typed=(variant == "exphormer")).to(dev)
    torch.manual_seed(1)
    q, k, v = (torch.randn(n, hl, hn, device=dev).mul(1.5).to(dtype).requires_grad_(True) for _ in range(3))
    etab = torch.randn(2, hl, hn, device=dev, requires_grad=True) if variant == "exphormer" else None
    dout = torch.randn(n, hl, hn, device=dev).to(dtype)
    out = edge_attention(q, k, v, g, variant=variant, etable=etab, dropout_p=dropout, dropout_seed=1234)
    out.backward(dout)
    got = [out.detach().float(), q.grad.float(), k.grad.float(), v.grad.float()]
    if etab is not None:
        got.append(etab.grad.float())
    q2, k2, v2 = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    e2 = etab.detach().clone().requires_grad_(True) if etab is not None else None
    ref = edge_attention_reference(q2, k2, v2, g, variant=variant, etable=e2, dropout_p=dropout, dropout_seed=1234)
    ref.backward(dout.float())
    want = [ref.detach(), q2.grad, k2.grad, v2.grad] + ([e2.grad] if e2 is not None else [])
    rtol, atol = TOL[dtype]
    names = ["out", "dq", "dk", "dv", "detab"]
    for name, a, b in zip(names, got, want):
        scale = max(1.0, float(b.abs().max()))
        err = float((a - b).abs().max())
        assert err <= atol * scale + rtol * scale, f"{variant}/{dtype}/{name}: max err {err} (scale {scale})"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hl,hn", [(8, 16), (1, 16), (4, 32), (2, 64), (3, 16), (1, 32)])
def test_edge_attention_plain(dtype, hl, hn):
    _run("plain", dtype, hl, hn)


@pytest.mark.parametrize("variant", ["gps", "exphormer"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_edge_attention_variants(variant, dtype):
    _run(variant, dtype, 4, 16)
    _run(variant, dtype, 1, 32)


def test_edge_attention_gps_dropout():
    _run("gps", torch.float32, 4, 16, dropout=0.4)
    _run("gps", torch.bfloat16, 2, 32, dropout=0.25)


@pytest.mark.parametrize("variant", ["plain", "gps", "exphormer"])
def test_edge_attention_hub_rows(variant):
    """A query with 5000 in-edges and a key used by 4000 queries are cut into work items of 64 edges."""
    _run(variant, torch.float32, 4, 16, hub_row=5000, hub_col=4000, n=4500, e=9000)
    _run(variant, torch.bfloat16, 1, 16, hub_row=20000, hub_col=3000, n=4500, e=9000)


@pytest.mark.parametrize("by_key", [False, True])
@pytest.mark.parametrize("dtype,hl,hn", [(torch.float32, 3, 8), (torch.bfloat16, 8, 16), (torch.float32, 4, 64), (torch.float16, 5, 128)])
def test_edge_attention_rows_around_the_work_item_edges(dtype, hl, hn, by_key):
    """Rows (queries, or keys of the backward pass) of 0 edges up to several reduction windows of 64 slots: one edge below, at
    and above the length from which a row is cut, whole and ragged last items, rows inside one window, ending at its end and
    running over several.  Rows wider than a warp (4 x 64 fp32, 5 x 128) take two head chunks.  Bit-equal when repeated."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    gen = torch.Generator().manual_seed(17)
    lengths = [0, 1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 320, 3000, 4096, 4097, 2, 12289, 130, 9000, 64 * 64 * 3]
    n = 700
    long_side = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths))
    other = torch.randint(0, n, (long_side.numel(),), generator=gen)
    ei = torch.stack([long_side, other] if by_key else [other, long_side])
    g = AttnGraph.from_edge_index(ei, n).to("cuda")
    q, k, v = (torch.randn(n, hl, hn, generator=gen).cuda().to(dtype).requires_grad_(True) for _ in range(3))
    dout = torch.randn(n, hl, hn, generator=gen).cuda().to(dtype)
    out = edge_attention(q, k, v, g)
    got = [out] + list(torch.autograd.grad(out, (q, k, v), dout))
    out2 = edge_attention(q, k, v, g)
    for a, b in zip(got, [out2] + list(torch.autograd.grad(out2, (q, k, v), dout))):
        assert torch.equal(a, b)
    q2, k2, v2 = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = edge_attention_reference(q2, k2, v2, g)
    rtol, atol = TOL[dtype]
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, [ref] + list(torch.autograd.grad(ref, (q2, k2, v2), dout.float()))):
        scale = max(1.0, float(b.abs().max()))
        assert float((a.float() - b).abs().max()) <= (atol + rtol) * scale, name


@pytest.mark.parametrize("variant,hl,hn", [("plain", 2, 16), ("plain", 1, 16), ("gps", 4, 16), ("exphormer", 2, 32)])
def test_edge_attention_routed_rows_match_local_rows(variant, hl, hn):
    """Routed stores on one GPU (the "destinations" are local buffers standing in for the peers' mappings): every context
    row also lands in its owner's slab, and routed dq / dk / dv rows equal the unrouted gradients - regular rows, a
    5,000-edge query row, a key used by 4,000 queries (split into work items), typed edges."""
    from budgetformer_b200.ops import _ext
    from budgetformer_b200.ops.edge_attention import _VARIANTS
    ext = _ext.load()
    dev = torch.device("cuda")
    torch.manual_seed(2)
    n_dest, rows_per = 4, 1200
    n = n_dest * rows_per
    g = random_attn_graph(n, 9000, hub_row=5000, hub_col=4000, seed=9, typed=(variant == "exphormer")).to(dev).ensure_transpose()
    w = hl * hn
    q, k, v = (torch.randn(n, hl, hn, device=dev).bfloat16() for _ in range(3))
    etab = (torch.randn(2, hl, hn, device=dev) * 0.5 + 1.0) if variant == "exphormer" else None
    vid = _VARIANTS[variant]
    src = 2                                                          # this "rank" is source 2 of 4
    out = torch.empty(n, hl, hn, device=dev, dtype=torch.bfloat16)
    z = torch.empty(n, hl, device=dev)
    slabs = [torch.full((n_dest * rows_per, w), 7.0, device=dev, dtype=torch.bfloat16) for _ in range(n_dest)]
    route = [rows_per, src * rows_per, w] + [t.data_ptr() for t in slabs]
    ext.edge_attn_fwd(q, k, v, out, z, g.rowptr, g.col, g.etype, etab, vid, 0.0, 0, -1, [], route)
    torch.cuda.synchronize()
    for d in range(n_dest):
        mine = slabs[d][src * rows_per:(src + 1) * rows_per]
        assert torch.equal(mine, out.view(n, w)[d * rows_per:(d + 1) * rows_per]), f"context rows of destination {d}"
        other = torch.cat([slabs[d][:src * rows_per], slabs[d][(src + 1) * rows_per:]])
        assert float((other - 7.0).abs().max()) == 0.0               # nobody else's slab was touched
    # backward: unrouted into a packed [n, ld] buffer, routed into slabs of the same row layout (k | v | q)
    ld = (3 * w + 63) // 64 * 64
    dout = torch.randn(n, hl, hn, device=dev).bfloat16()
    def grads(route):
        buf = torch.full((n, ld), 3.0, device=dev, dtype=torch.bfloat16)
        part = lambda i: buf[:, i * w:(i + 1) * w].view(n, hl, hn)
        zd = torch.empty(n, hl, 2, device=dev)
        detab = torch.zeros(2, hl, hn, device=dev) if etab is not None else None
        ext.edge_attn_bwd(q, k, v, out, z, dout, part(2), part(0), part(1), zd, g.rowptr, g.col, g.etype, g.t_rowptr, g.t_row,
                          g.t_eid, etab, detab, vid, 0.0, 0, -1, g.t_task, g.t_split, int(g.kv_slots), [], route)
        torch.cuda.synchronize()
        return buf
    plain = grads([])
    gslabs = [torch.full((n_dest * rows_per, ld), 5.0, device=dev, dtype=torch.bfloat16) for _ in range(n_dest)]
    untouched = grads([rows_per, src * rows_per, ld, 2 * w, 0, w] + [t.data_ptr() for t in gslabs])
    assert float((untouched - 3.0).abs().max()) == 0.0               # routed gradients never touch the local buffer
    for d in range(n_dest):
        got = gslabs[d][src * rows_per:(src + 1) * rows_per, :3 * w]
        want = plain[d * rows_per:(d + 1) * rows_per, :3 * w]
        # (the 5,000-edge query row adds its dq partials with atomics: last-bit differences between two runs)
        assert torch.allclose(got.float(), want.float(), atol=2e-2, rtol=2e-2), f"gradient rows of destination {d}"
        if 3 * w < ld:                                               # the padding columns of a packed row stay untouched
            assert float((gslabs[d][src * rows_per:(src + 1) * rows_per, 3 * w:] - 5.0).abs().max()) == 0.0
        other = torch.cat([gslabs[d][:src * rows_per], gslabs[d][(src + 1) * rows_per:]])
        assert float((other - 5.0).abs().max()) == 0.0
    # a route that does not cover the rows is refused before anything is launched
    with pytest.raises(RuntimeError):
        ext.edge_attn_fwd(q, k, v, out, z, g.rowptr, g.col, g.etype, etab, vid, 0.0, 0, -1, [], [rows_per + 1, 0, w] + [t.data_ptr() for t in slabs])


def test_edge_attention_strided_qkv_views():
    dev = torch.device("cuda")
    n, hl, hn = 300, 4, 16
    g = random_attn_graph(n, 2000, seed=3).to(dev)
    qkv = torch.randn(n, 3, hl, hn, device=dev, dtype=torch.bfloat16)
    q, k, v = qkv[:, 0], qkv[:, 1], qkv[:, 2]
    out = edge_attention(q, k, v, g)
    ref = edge_attention_reference(q.float(), k.float(), v.float(), g)
    assert torch.allclose(out.float(), ref, atol=3e-2, rtol=3e-2)


def test_edge_attention_empty_rows_and_determinism():
    dev = torch.device("cuda")
    n, hl, hn = 128, 2, 16
    g = random_attn_graph(n, 100, seed=5).to(dev)          # most queries have no in-edges
    q, k, v = (torch.randn(n, hl, hn, device=dev, dtype=torch.bfloat16) for _ in range(3))
    a = edge_attention(q, k, v, g)
    b = edge_attention(q, k, v, g)
    assert torch.equal(a, b)
    deg = (g.rowptr[1:] - g.rowptr[:-1])
    assert float(a[deg == 0].abs().max()) == 0.0


@pytest.mark.parametrize("exph", [False, True])
@pytest.mark.parametrize("cfg", [(4, 4, 2, 4), (2, 6, 3, 5), (8, 0, 2, 4), (0, 5, 2, 3), (32, 32, 8, 8), (16, 16, 4, 6)])
def test_gpu_builder_matches_cpu_builder(cfg, exph):
    br, bw, w, l = cfg
    topo, _ = random_topology(700, 6000, hub_in=900, hub_out=400, seed=11)
    cpu = build_attn_graph(topo, br, bw, w, l, 77, exphormer=exph)
    gpu = build_attn_graph(topo.to("cuda"), br, bw, w, l, 77, exphormer=exph)
    assert torch.equal(cpu.rowptr, gpu.rowptr.cpu())
    assert torch.equal(cpu.col, gpu.col.cpu())
    if exph:
        assert torch.equal(cpu.etype, gpu.etype.cpu())
    assert cpu._totals.tolist() == gpu._totals.cpu().tolist()


@pytest.mark.parametrize("exph", [False, True])
@pytest.mark.parametrize("cfg", [(4, 4, 2, 4), (8, 8, 2, 4), (32, 16, 4, 6), (1, 0, 2, 4)])
def test_gpu_builder_ranks_long_rows_with_a_block_per_row(cfg, exph, monkeypatch):
    """Queries with more in-edges than the block threshold (one of 30,000 with many repeated sources, one just above
    the threshold, one just below it) are ranked by a thread block each: same graph as the CPU builder, as the device
    builder with the pre-pass switched off, and as a build of row ranges that cut between the long rows."""
    from budgetformer_b200.ops import _ext
    br, bw, w, l = cfg
    thr = int(_ext.load().BUILD_HUB_DEGREE)
    g = torch.Generator().manual_seed(5)
    n = 3000
    ei = torch.randint(0, n, (2, 20000), generator=g)
    extra = [torch.stack([torch.randint(0, 500, (30000,), generator=g), torch.full((30000,), 0)]),
             torch.stack([torch.randint(0, n, (thr + 1,), generator=g), torch.full((thr + 1,), 1700)]),
             torch.stack([torch.randint(0, n, (thr - 30,), generator=g), torch.full((thr - 30,), 2999)])]
    topo = Topology.from_edge_index(torch.cat([ei] + extra, 1), n)
    dev = topo.to("cuda")
    assert dev.in_hub_rows(thr).tolist() == [0, 1700]
    cpu = build_attn_graph(topo, br, bw, w, l, 91, exphormer=exph)
    gpu = build_attn_graph(dev, br, bw, w, l, 91, exphormer=exph)
    assert torch.equal(cpu.rowptr, gpu.rowptr.cpu()) and torch.equal(cpu.col, gpu.col.cpu())
    if exph:
        assert torch.equal(cpu.etype, gpu.etype.cpu())
    assert cpu._totals.tolist() == gpu._totals.cpu().tolist()
    # row ranges (what one rank of a sharded build selects): [0, 1500) holds the first long row, [1500, 3000) the second
    ext = _ext.load()
    cap = max(br + bw + (1 if exph else 0), 1)
    cols, cnts = [], []
    for begin in (0, 1500):
        ell_col = torch.empty(1500 * cap, dtype=torch.int32, device="cuda")
        ell_cnt = torch.empty(1500, dtype=torch.int32, device="cuda")
        ell_typ = torch.empty(1500 * cap, dtype=torch.uint8, device="cuda") if exph else None
        totals = torch.zeros(2, dtype=torch.int64, device="cuda")
        ext.budget_select_rows(dev.in_rowptr, dev.in_src, dev.out_rowptr, dev.out_col, n, br, bw, w, l, exph, 91, begin, 1500,
                               ell_col, ell_cnt, ell_typ, totals, dev.in_hub_rows(thr))
        cols.append(ell_col); cnts.append(ell_cnt)
    rowptr, col, _ = ext.ell_rows_to_csr(torch.cat(cols), torch.cat(cnts), None, n, cap)
    assert torch.equal(rowptr.cpu(), cpu.rowptr) and torch.equal(col.cpu(), cpu.col)
    monkeypatch.setenv("BF_BUILD_HUB_BLOCKS", "0")
    plain = build_attn_graph(dev, br, bw, w, l, 91, exphormer=exph)
    assert torch.equal(plain.col, gpu.col) and torch.equal(plain.rowptr, gpu.rowptr)


@pytest.mark.parametrize("exph", [False, True])
@pytest.mark.parametrize("cfg", [(0, 4, 1, 1), (4, 0, 2, 4), (3, 5, 3, 5), (8, 9, 5, 7), (16, 16, 2, 16), (17, 32, 7, 6)])
def test_gpu_builder_at_the_edges_of_its_lists(cfg, exph):
    """List lengths 4, 8, 16 and 32, odd walk counts, a last block of one thread, and rows around the lengths at which a thread, the
    warp and a cluster of blocks rank them; rows whose sources repeat (their hashes come in lumps, so the estimated bound lets far too
    few or too many pass) and rows without edges."""
    br, bw, w, l = cfg
    g = torch.Generator().manual_seed(7)
    n = 128 * 9 + 1
    degs = [0, 1, 2, 31, 32, 33, 34, 63, 64, 65, 127, 128, 129, 130, 4095, 4096, 4097, 9000]
    rows = [torch.stack([torch.randint(0, n, (d,), generator=g), torch.full((d,), 3 + 7 * i)]) for i, d in enumerate(degs)]
    rows += [torch.stack([torch.randint(0, few, (d,), generator=g), torch.full((d,), 600 + 5 * i)])
             for i, (few, d) in enumerate([(1, 40), (2, 100), (5, 200), (3, 4090), (1, 5000), (4, 8200), (40, 300)])]
    rows.append(torch.randint(0, n, (2, 4000), generator=g))
    topo = Topology.from_edge_index(torch.cat(rows, 1), n)
    cpu = build_attn_graph(topo, br, bw, w, l, 13, exphormer=exph)
    gpu = build_attn_graph(topo.to("cuda"), br, bw, w, l, 13, exphormer=exph)
    assert torch.equal(cpu.rowptr, gpu.rowptr.cpu()) and torch.equal(cpu.col, gpu.col.cpu())
    if exph:
        assert torch.equal(cpu.etype, gpu.etype.cpu())
    assert cpu._totals.tolist() == gpu._totals.cpu().tolist()


@pytest.mark.parametrize("exph", [False, True])
@pytest.mark.parametrize("n", [1200, 30001, 66001])
@pytest.mark.parametrize("cfg", [(4, 4, 2, 4), (8, 8, 8, 8), (7, 3, 3, 5), (2, 8, 1, 16), (8, 8, 11, 4), (3, 12, 5, 7), (16, 16, 33, 3), (25, 4, 2, 4), (32, 32, 3, 6), (32, 0, 0, 0)])
def test_gpu_builder_forms(cfg, n, exph):
    """Eight lanes or a warp per query (few queries for their walks), a thread with eight walks or two under way; long rows among short ones (the warp
    ranks them), warps whose rows are all of medium length (their lanes do), and rows of up to 4,096 edges at the largest budgets, where
    hashes fill the estimated bound's slots now and then."""
    br, bw, w, l = cfg
    g = torch.Generator().manual_seed(br + w)
    at, rows = 0, []
    for i in range(64):                                   # two warps of 33 to 110 edges, one of mixed lengths
        rows.append((at + i, 33 + i * 5 % 78))
    for i, d in enumerate([500, 3, 4096, 40, 0, 70, 31, 33, 1500, 700, 4000, 2, 900, 1000, 1100, 1200, 1300]):
        rows.append((96 + i, d))
    dst = torch.repeat_interleave(torch.tensor([r for r, _ in rows]), torch.tensor([d for _, d in rows]))
    ei = torch.stack([torch.randint(0, n, (dst.numel(),), generator=g), dst])
    topo = Topology.from_edge_index(torch.cat([ei, torch.randint(0, n, (2, 3000), generator=g)], 1), n)
    cpu = build_attn_graph(topo, br, bw, w, l, 29, exphormer=exph)
    gpu = build_attn_graph(topo.to("cuda"), br, bw, w, l, 29, exphormer=exph)
    assert torch.equal(cpu.rowptr, gpu.rowptr.cpu()) and torch.equal(cpu.col, gpu.col.cpu())
    if exph:
        assert torch.equal(cpu.etype, gpu.etype.cpu())
    assert cpu._totals.tolist() == gpu._totals.cpu().tolist()


def test_gpu_builder_seed_changes_graph_and_is_reproducible():
    topo, _ = random_topology(500, 5000, seed=2)
    t = topo.to("cuda")
    a = build_attn_graph(t, 4, 4, 2, 4, 1)
    b = build_attn_graph(t, 4, 4, 2, 4, 1)
    c = build_attn_graph(t, 4, 4, 2, 4, 2)
    assert torch.equal(a.col, b.col) and torch.equal(a.rowptr, b.rowptr)
    assert not (a.col.numel() == c.col.numel() and torch.equal(a.col, c.col))


def test_extension_is_loaded_from_tree():
    from budgetformer_b200.ops import _ext
    mod = _ext.load()
    assert "budgetformer_b200/csrc/build" in mod.__file__.replace("\\", "/")


@pytest.mark.parametrize("hub", [False, True])
def test_device_transpose_matches_torch_path(hub):
    """csrc/graph_transpose.cu (radix sort over node-id bits + compaction) gives the same by-key view and the same
    dK/dV work list as the PyTorch construction used for CPU graphs."""
    from budgetformer_b200.graph.attn_graph import AttnGraph, add_virtual_node
    n = 5000
    g = random_attn_graph(n, 30000, hub_col=700, seed=3)
    if hub:
        g = add_virtual_node(g, n, n)                     # row 0 holds every node; key 0 is used by every query
    ref = AttnGraph(g.num_rows, g.rowptr.cpu(), g.col.cpu(), None).ensure_transpose()
    dev = AttnGraph(g.num_rows, g.rowptr.cuda(), g.col.cuda(), None).ensure_transpose()
    for name in ("t_rowptr", "t_row", "t_eid", "t_task", "t_split"):
        a, b = getattr(ref, name), getattr(dev, name).cpu()
        assert a.shape == b.shape and torch.equal(a.to(b.dtype), b), name
    assert ref.kv_slots == dev.kv_slots
    if hub:
        assert dev.kv_slots > 0 and dev.t_split.size(0) >= 1


@pytest.mark.parametrize("longest", [64, 65, 4000, 8100])
def test_device_transpose_of_one_longer_row(longest):
    """Blocks of 256 rows with at most 8,192 edges: rows up to 64 are marked by their threads, one longer sends its block another way.
    The last block holds one row."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    g = torch.Generator().manual_seed(longest)
    n = 256 * 3 + 1
    deg = torch.randint(0, 20, (n,), generator=g)
    deg[256:512] = 0
    deg[300], deg[511], deg[n - 1] = longest, 60, longest
    dst = torch.repeat_interleave(torch.arange(n), deg)
    ref = AttnGraph.from_edge_index(torch.stack([torch.randint(0, n, (dst.numel(),), generator=g), dst]), n).ensure_transpose()
    dev = AttnGraph(n, ref.rowptr.cuda(), ref.col.cuda(), None).ensure_transpose()
    for name in ("t_rowptr", "t_row", "t_eid"):
        a, b = getattr(ref, name), getattr(dev, name).cpu()
        assert torch.equal(a.to(b.dtype), b), name


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_batch_norm_kernels_match_pytorch(dtype):
    """Forward, running statistics and all three gradients of the row BatchNorm against nn.BatchNorm1d in fp32."""
    from budgetformer_b200.ops.norm import batch_norm
    torch.manual_seed(0)
    rows, h = 5003, 64
    x = (torch.randn(rows, h, device="cuda") * 1.7 + 0.6).to(dtype)
    bn = torch.nn.BatchNorm1d(h).cuda()
    ref = torch.nn.BatchNorm1d(h).cuda()
    with torch.no_grad():
        bn.weight.uniform_(0.5, 1.5); bn.bias.uniform_(-0.5, 0.5)
        ref.weight.copy_(bn.weight); ref.bias.copy_(bn.bias)
    xa = x.clone().requires_grad_(True)
    xb = x.float().clone().requires_grad_(True)
    g = torch.randn(rows, h, device="cuda")
    for _ in range(2):                                   # second call uses a non-zero running mean as the shift
        ya = batch_norm(xa, bn)
        yb = ref(xb)
    (ya.float() * g).sum().backward()
    (yb * g).sum().backward()
    tol = 3e-2 if dtype == torch.bfloat16 else 1e-4
    assert ya.dtype == dtype and (ya.float() - yb).abs().max() < tol
    assert (bn.running_mean - ref.running_mean).abs().max() < 1e-3
    assert (bn.running_var - ref.running_var).abs().max() < 2e-3
    scale = xb.grad.abs().max()
    assert (xa.grad.float() - xb.grad).abs().max() < (4e-2 if dtype == torch.bfloat16 else 1e-4) * max(1.0, float(scale))
    ptol = 2e-2 if dtype == torch.bfloat16 else 2e-3
    assert (bn.weight.grad - ref.weight.grad).abs().max() < ptol * ref.weight.grad.abs().max() + 5e-2
    assert (bn.bias.grad - ref.bias.grad).abs().max() < ptol * ref.bias.grad.abs().max() + 5e-2
    bn.eval(); ref.eval()
    assert (batch_norm(x, bn).float() - ref(x.float())).abs().max() < tol


@pytest.mark.parametrize("h,affine,momentum,track,stats", [
    (8, True, 0.1, True, torch.float32), (128, True, 0.3, True, torch.float32), (136, False, 0.1, True, torch.float32),
    (64, True, None, True, torch.float32), (64, True, 0.1, False, torch.float32), (64, True, 0.1, True, torch.float64)])
def test_batch_norm_coefficients_by_one_launch(h, affine, momentum, track, stats):
    """Every form of the module: columns up to and past a block of the coefficient kernel, no affine part, a cumulative average, no
    running statistics, running statistics of another type (these three move outside the kernel)."""
    from budgetformer_b200.ops.norm import batch_norm
    make = lambda: torch.nn.BatchNorm1d(h, affine=affine, momentum=momentum, track_running_stats=track)
    gen = torch.Generator(device="cuda").manual_seed(h)
    bn, ref = make().cuda(), make().cuda().double()
    if track:
        bn.running_mean, bn.running_var = bn.running_mean.to(stats), bn.running_var.to(stats)
    for step in range(3):
        x = torch.randn(1009, h, generator=gen, device="cuda") * 2 + 1 + step
        xa, xb = x.clone().requires_grad_(), x.double().requires_grad_()
        g = torch.randn(1009, h, generator=gen, device="cuda")
        version = bn.running_mean._version if track else 0
        ya, yb = batch_norm(xa, bn), ref(xb)
        ya.backward(g); yb.backward(g.double())
        # fp32 sums of 10^3 terms of size 1 to 10: 1e-5 of the result's scale
        assert (ya - yb).abs().max() <= 1e-5 * yb.abs().max()
        assert (xa.grad - xb.grad).abs().max() <= 1e-5 * xb.grad.abs().max()
        if track:
            assert int(bn.num_batches_tracked) == step + 1 and bn.running_mean._version > version
            assert (bn.running_mean - ref.running_mean).abs().max() <= 1e-5 and (bn.running_var - ref.running_var).abs().max() <= 1e-4
    bn.eval(), ref.eval()
    with torch.no_grad():
        ya, yb = batch_norm(x, bn), ref(x.double())
    assert ya.dtype == x.dtype and (ya - yb).abs().max() <= 3e-5 * yb.abs().max()       # the running statistics' 1e-5 as well


@pytest.mark.parametrize("rows,momentum", [(1, 0.1), (2, 0.3), (3001, 0.1)])
def test_batch_norm_coefficients_equal_the_operators(rows, momentum):
    """The coefficient kernels give what PyTorch's operators give, bit for bit: a single row and a constant column have no variance,
    however large their mean."""
    from budgetformer_b200.ops import _ext
    ext, h = _ext.load(), 64
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, h, generator=g, device="cuda") * 10 ** torch.linspace(-3, 4.5, h, device="cuda")
    x[:, 5] = 29952.0
    x[:, 6] = 12345.67
    shift, w, b = (torch.randn(h, generator=g, device="cuda") for _ in range(3))
    n, eps = torch.full((1,), float(rows), device="cuda"), 1e-5      # on the device: a division by a host number is a multiplication
    s1, s2 = (x - shift).sum(0), ((x - shift) ** 2).sum(0)
    run_mean, run_var = shift.clone(), torch.rand(h, generator=g, device="cuda")
    m1 = s1 / n
    var = (s2 / n - m1 * m1).clamp_min(0.0)
    mean = m1 + shift
    rstd = torch.rsqrt(var + eps)
    a = w * rstd
    want = [mean, var, rstd, a, b - mean * a, run_mean.mul(1 - momentum).add(mean, alpha=momentum),
            run_var.mul(1 - momentum).add(var * (n / (n - 1.0).clamp(min=1.0)), alpha=momentum)]
    got = list(ext.bn_finish(s1, s2, None, float(rows), shift, w, b, eps, run_mean, run_var, momentum, None).unbind(0)) + [run_mean, run_var]
    for i, (p, q) in enumerate(zip(got, want)):
        assert torch.equal(p, q), i
    if rows == 1:
        assert not got[1].any()
    sb, sg = (torch.randn(h, generator=g, device="cuda") * rows for _ in range(2))
    want = [a, -a * rstd * (sg / n), a * (-(sb / n) + mean * rstd * (sg / n))]
    for p, q in zip(ext.bn_bwd_finish(sb, sg, None, float(rows), mean, rstd, w).unbind(0), want):
        assert torch.equal(p, q)


def test_batch_norm_coefficients_with_the_count_on_the_device():
    """What a statistics group gives: sums and a number of rows that only the device knows."""
    from budgetformer_b200.ops import _ext
    ext, h = _ext.load(), 72
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, dy = (torch.randn(500, h, generator=gen, device="cuda") for _ in range(2))
    count = torch.tensor([500.0], device="cuda")
    for dev, host in ((count, 0.0), (None, 500.0)):
        mean, var, rstd, a, b = ext.bn_finish(x.sum(0), (x * x).sum(0), dev, host, None, None, None, 1e-5, None, None, 0.0, None).unbind(0)
        ref = x.double()
        want = torch.nn.functional.batch_norm(ref, None, None, training=True, eps=1e-5)
        assert (mean - ref.mean(0)).abs().max() < 1e-6 and (var - ref.var(0, unbiased=False)).abs().max() < 1e-5
        assert (x * a + b - want).abs().max() < 1e-5
        sb, sg = dy.sum(0), (dy * (x - mean) * rstd).sum(0)
        a, b, c0 = ext.bn_bwd_finish(sb, sg, dev, host, mean, rstd, None).unbind(0)
        xr = ref.requires_grad_()
        torch.nn.functional.batch_norm(xr, None, None, training=True, eps=1e-5).backward(dy.double())
        assert (dy * a + x * b + c0 - xr.grad).abs().max() < 1e-5


@pytest.mark.parametrize("variant", ["plain", "gps", "exphormer"])
def test_edge_attention_kernels_against_coo_oracle(variant):
    """Forward and backward of the CUDA kernels against the float32 oracle written on the reference's COO layout
    (hub row and hub key included)."""
    from budgetformer_b200 import oracle
    from tests.helpers import random_attn_graph
    torch.manual_seed(12)
    n, h, hn = 700, 4, 16
    g = random_attn_graph(n, 5000, hub_row=1500, hub_col=1400, seed=8, typed=variant == "exphormer").to("cuda")
    ei = g.edge_index()
    q, k, v = (torch.randn(n, h, hn, device="cuda", requires_grad=True) for _ in range(3))
    emb = torch.randn(2, h * hn, device="cuda")
    proj = torch.randn(h * hn, h * hn, device="cuda") * 0.1
    table = (emb @ proj.t()).view(2, h, hn) if variant == "exphormer" else None
    out = edge_attention(q, k, v, g, variant=variant, etable=table)
    if variant == "plain":
        ref = oracle.attention.sparse_attention(q, k, v, ei)
    elif variant == "gps":
        ref = oracle.attention.gps_attention(q, k, v, ei)
    else:
        ref = oracle.attention.exphormer_attention(q, k, v, ei, emb, proj)
    assert torch.allclose(out, ref, atol=2e-4, rtol=2e-4), float((out - ref).abs().max())
    dout = torch.randn_like(out)
    got = torch.autograd.grad(out, (q, k, v), dout)
    want = torch.autograd.grad(ref, (q, k, v), dout)
    for a, b, name in zip(got, want, "qkv"):
        assert torch.allclose(a, b, atol=5e-4, rtol=1e-3), (name, float((a - b).abs().max()))


def test_edge_attention_with_understated_degree_bound():
    """``max_degree`` is a hint from the graph builder.  A hint below the true maximum must not drop edges: rows longer
    than the hint are either walked by the regular kernels (no hub list) or by hub blocks that stride over their chunks."""
    from tests.helpers import random_attn_graph
    torch.manual_seed(3)
    n, hl, hn = 3000, 2, 16
    g = random_attn_graph(n, 6000, hub_row=20000, hub_col=2500, seed=5).to("cuda")
    q, k, v = (torch.randn(n, hl, hn, device="cuda") for _ in range(3))
    ref = edge_attention_reference(q, k, v, g)
    for wrong in (8, 1500):                     # below the hub threshold (no hub list at all) / above it but far too small
        g.max_degree = wrong
        qq, kk, vv = (t.clone().requires_grad_(True) for t in (q, k, v))
        out = edge_attention(qq, kk, vv, g)
        assert torch.allclose(out, ref, atol=2e-4, rtol=2e-4), (wrong, float((out - ref).abs().max()))
        out.sum().backward()
        q2, k2, v2 = (t.clone().requires_grad_(True) for t in (q, k, v))
        edge_attention_reference(q2, k2, v2, g).sum().backward()
        for a, b in ((qq, q2), (kk, k2), (vv, v2)):
            assert torch.allclose(a.grad, b.grad, atol=1e-3, rtol=1e-3), wrong
