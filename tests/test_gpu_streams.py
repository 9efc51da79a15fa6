"""Edge attention as streams of segments, the fp32 weight gradient and the row-wise element kernels, at the sizes where their
splits end: one row, partial warps, heads that do not fill a lane group, several segments per lane group, empty rows."""
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


def _graph_of(edges, n):
    from budgetformer_b200.graph.attn_graph import AttnGraph
    return AttnGraph.from_edge_index(edges, n).to("cuda")


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
    (30011, 8, 32, 8, torch.bfloat16), (30011, 8, 8, 6, torch.float16), (9001, 4, 64, 8, torch.float32),
    # two and three segments a lane group in every pass, and the most that one takes (8; 32 in the typed dQ pass)
    (35003, 8, 32, 5, torch.bfloat16), (25013, 4, 64, 5, torch.float32), (134999, 8, 32, 4, torch.bfloat16),
    (310007, 4, 64, 3, torch.float16),
    # behind the lines up to which the forward pass walks rows without a stream (k and v of 200 MB; 100 MB with heads of 8)
    (101021, 4, 64, 3, torch.float32), (1600007, 2, 16, 3, torch.bfloat16), (410003, 8, 8, 3, torch.float16),
    (5003, 8, 8, 9, torch.float32)])
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
    # Row by row, since one wrong row among thousands is what a wrong segment end looks like.  16 bits: the context is rounded when
    # stored (unit 2^-9 / 2^-12) and D = <dout, out> inherits it; fp32: sums of <= 10^3 terms.  Score gradients are differences
    # <dout, v_j> - D that cancel (to zero in a row of one edge): what the rounding of D leaves is at most
    # unit * |dout_i| |out_i| |k_j| / sqrt(hn) an edge, of the order of unit * |dout_i|: the second term, for a key once per query.
    tol = {torch.float32: 2e-5, torch.float16: 4e-3, torch.bfloat16: 2.5e-2}[dtype]
    rows = lambda t: t.double().flatten(1).norm(dim=1)
    per_key = torch.bincount(graph.col.long(), minlength=n).double().clamp(min=1).sqrt() * heads ** 0.5 * hn ** 0.5
    for i, (a, b) in enumerate(zip(got[:4], want[:4])):
        err, size = rows(a.double() - b.double()), rows(b) + (rows(dout) if i < 2 else per_key)
        worst = int((err / size).argmax())
        assert bool((err <= tol * size + 1e-6).all()), (i, worst, float(err[worst]), float(size[worst]))
    for a, b in zip(got[4:], want[4:]):                                    # the type table's gradient: sums over all rows
        assert float((a.double() - b.double()).norm()) <= tol * (float(b.double().norm()) + float(dout.double().norm())) + 1e-6


@pytest.mark.parametrize("bounded", [True, False])
@pytest.mark.parametrize("variant", ["plain", "gps", "exphormer"])
@pytest.mark.parametrize("heads,hn,dtype", [(8, 16, torch.bfloat16), (3, 32, torch.float16), (5, 64, torch.bfloat16), (1, 128, torch.bfloat16),
                                            (32, 8, torch.float16), (4, 16, torch.float32), (12, 16, torch.bfloat16), (2, 128, torch.float32)])
def test_attention_chunks_of_edges(heads, hn, dtype, variant, bounded):
    """Query rows and keys of 0 to 70 edges: one edge less than a lane group's chunk of the list, the chunk and one more, for groups of
    every width, between empty ones.  With a known bound on the rows (streams) and without (a warp of one row)."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    n = 1130
    gen = torch.Generator().manual_seed(heads + hn)
    deg = torch.where(torch.arange(n) % 8 == 1, torch.arange(n) % 71, torch.zeros((), dtype=torch.long))
    a = torch.repeat_interleave(torch.arange(n), deg)
    b = torch.randint(0, n, (a.numel(),), generator=gen)
    edges = torch.cat([torch.stack([a, b]), torch.stack([b, a])], 1)
    if variant == "exphormer":
        edges = torch.cat([edges, torch.randint(0, 2, (1, edges.size(1)), generator=gen)])
    graph = AttnGraph.from_edge_index(edges, n).to("cuda")
    if bounded:
        graph.max_degree = int((graph.rowptr[1:] - graph.rowptr[:-1]).max())
        assert graph.max_degree <= 128 and graph.num_edges < 12 * n          # what keeps 16-bit rows on the streams
    gen = torch.Generator(device="cuda").manual_seed(hn)
    q, k, v, dout = (torch.randn(n, heads, hn, generator=gen, device="cuda").to(dtype) for _ in range(4))
    tab = torch.randn(2, heads, hn, generator=gen, device="cuda") if variant == "exphormer" else None
    p = 0.3 if variant == "gps" else 0.0
    want = _reference(q, k, v, dout, graph, tab, variant, p, 5)
    args = [x.requires_grad_() for x in (q, k, v)] + ([tab.requires_grad_()] if tab is not None else [])
    out = edge_attention(q, k, v, graph, variant=variant, etable=tab, dropout_p=p, dropout_seed=5)
    got = [out] + list(torch.autograd.grad(out, args, dout))
    # bounds as in test_attention_streams
    tol = {torch.float32: 2e-5, torch.float16: 4e-3, torch.bfloat16: 2.5e-2}[dtype]
    rows = lambda t: t.double().flatten(1).norm(dim=1)
    per_key = torch.bincount(graph.col.long(), minlength=n).double().clamp(min=1).sqrt() * heads ** 0.5 * hn ** 0.5
    for i, (x, y) in enumerate(zip(got[:4], want[:4])):
        assert bool((rows(x.double() - y.double()) <= tol * (rows(y) + (rows(dout) if i < 2 else per_key)) + 1e-6).all()), i
    for x, y in zip(got[4:], want[4:]):
        assert float((x.double() - y.double()).norm()) <= tol * (float(y.double().norm()) + float(dout.double().norm())) + 1e-6


@pytest.mark.parametrize("heads,hn,dtype", [(3, 8, torch.float16), (5, 64, torch.bfloat16), (2, 128, torch.float32), (9, 16, torch.float32)])
def test_sums_of_cut_rows(heads, hn, dtype):
    """Query rows and keys of two slots (of 64 edges) to several windows (of 64 slots), with eight slots and nine among them, side by side so
    that windows start and end inside them; widths below, at and off a warp's 128 columns."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    degs = torch.tensor([129, 512, 513, 576, 577, 0, 5, 1000, 4096, 4160, 130, 200, 8200, 640, 150, 3, 129, 600] + [140] * 30)
    n, gen = 1200, torch.Generator().manual_seed(heads)
    a = torch.repeat_interleave(torch.arange(len(degs)), degs)
    b = torch.randint(100, n, (a.numel(),), generator=gen)
    graph = AttnGraph.from_edge_index(torch.cat([torch.stack([a, b]), torch.stack([b, a])], 1), n).to("cuda")
    gen = torch.Generator(device="cuda").manual_seed(hn)
    q, k, v, dout = (torch.randn(n, heads, hn, generator=gen, device="cuda").to(dtype) for _ in range(4))
    want = _reference(q, k, v, dout, graph, None, "plain", 0.0, 0)
    args = [x.requires_grad_() for x in (q, k, v)]
    out = edge_attention(*args, graph)
    got = [out] + list(torch.autograd.grad(out, args, dout))
    # bounds as in test_attention_streams, with the fp32 sums' share for rows of 8 k terms
    tol = {torch.float32: 4e-5, torch.float16: 4e-3, torch.bfloat16: 2.5e-2}[dtype]
    rows = lambda t: t.double().flatten(1).norm(dim=1)
    per_key = torch.bincount(graph.col.long(), minlength=n).double().clamp(min=1).sqrt() * heads ** 0.5 * hn ** 0.5
    for i, (x, y) in enumerate(zip(got, want)):
        assert bool((rows(x.double() - y.double()) <= tol * (rows(y) + (rows(dout) if i < 2 else per_key)) + 1e-6).all()), i


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,hn", [(1, 8), (1, 16), (1, 32), (2, 16), (4, 8)])
def test_narrow_rows_keep_the_precision_of_dq(heads, hn, dtype):
    """Rows of 16 to 64 bytes: dQ against 64 bits is as far off as storing the context and the result in 16 bits makes it (D takes
    the rounded context), and no further.  dout / (Z + eps) rounded to 16 bits instead of dout gives 1.5 times that."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    n, deg = 6007, 6
    gen = torch.Generator(device="cuda").manual_seed(hn + heads)
    dst = torch.arange(n, device="cuda").repeat_interleave(deg)
    src = torch.randint(0, n, (n * deg,), generator=gen, device="cuda")
    graph = AttnGraph.from_edge_index(torch.stack([src, dst]), n)
    q, k, v, dout = (torch.randn(n, heads, hn, generator=gen, device="cuda").to(dtype) for _ in range(4))
    args = [t.requires_grad_() for t in (q, k, v)]
    out = edge_attention(*args, graph)
    dq = torch.autograd.grad(out, q, dout)[0].double()

    kd, vd, g = k.detach().double()[src].view(n, deg, heads, hn), v.detach().double()[src].view(n, deg, heads, hn), dout.double()
    s = torch.einsum("nhd,nehd->neh", q.detach().double(), kd) / hn ** 0.5
    w = s.clamp(-5, 5).exp()
    p = w / (w.sum(1, keepdim=True) + 1e-6)
    ctx = torch.einsum("neh,nehd->nhd", p, vd)

    def grad(c):
        ds = p * (torch.einsum("nhd,nehd->neh", g, vd) - (g * c).sum(-1)[:, None]) * (s.abs() < 5)
        return torch.einsum("neh,nehd->nhd", ds, kd) / hn ** 0.5

    want = grad(ctx)
    least = float((grad(ctx.to(dtype).double()).to(dtype).double() - want).norm())
    assert float((dq - want).norm()) <= 1.2 * least, (float((dq - want).norm()) / least, least / float(want.norm()))


@pytest.mark.parametrize("virtual_node", [False, True])
def test_lists_of_a_graph_serve_every_stream(virtual_node):
    """The lists that a graph makes of itself on first use are complete when the host gets them (nothing is queued behind the read
    of their length), so another stream may use them at once; forward and backward on two streams, one after the other."""
    from budgetformer_b200.graph.attn_graph import AttnGraph, add_virtual_node
    from budgetformer_b200.ops.edge_attention import edge_attention
    graph = _graph(4001, 300, 5, False)
    if virtual_node:
        graph.max_degree = 300
        graph = add_virtual_node(graph, 4001, 4001)
    fresh = AttnGraph(graph.num_rows, graph.rowptr, graph.col)
    torch.cuda.synchronize()
    fresh.long_rows()
    assert torch.cuda.current_stream().query()
    fresh.ensure_transpose()
    assert torch.cuda.current_stream().query()
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, dout = (torch.randn(graph.num_rows, 4, 16, generator=gen, device="cuda") for _ in range(4))
    want = _reference(q, k, v, dout, graph, None, "plain", 0.0, 0)
    args = [t.requires_grad_() for t in (q, k, v)]
    torch.cuda.synchronize()
    got = []
    for _ in range(2):
        with torch.cuda.stream(torch.cuda.Stream()):
            out = edge_attention(*args, graph)
            got.append([out] + list(torch.autograd.grad(out, args, dout)))
    torch.cuda.synchronize()
    assert len({s for kind, s in graph._list_users if kind == "long"}) == 2
    for res in got:
        for a, b in zip(res, want):
            assert float((a.double() - b.double()).norm()) <= 2e-5 * (float(b.double().norm()) + float(dout.norm()))


def test_virtual_node_beside_a_row_above_its_declared_bound():
    """add_virtual_node lists the virtual node's row without looking at the others; a row that is longer than the graph's degree
    bound says is walked all the same."""
    from budgetformer_b200.graph.attn_graph import add_virtual_node
    from budgetformer_b200.ops.edge_attention import edge_attention
    graph = _graph(1500, 300, 9, False)
    graph.max_degree = 8
    graph = add_virtual_node(graph, 1500, 1500)
    assert graph.q_task is not None and int(graph.q_task.size(0)) == 24 and graph.q_split.tolist() == [[0, 0, 24]]
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, dout = (torch.randn(1501, 2, 16, generator=gen, device="cuda") for _ in range(4))
    want = _reference(q, k, v, dout, graph, None, "plain", 0.0, 0)
    args = [t.requires_grad_() for t in (q, k, v)]
    out = edge_attention(*args, graph)
    for a, b in zip([out] + list(torch.autograd.grad(out, args, dout)), want):
        assert float((a.double() - b.double()).norm()) <= 2e-5 * (float(b.double().norm()) + float(dout.norm()))


@pytest.mark.parametrize("listed_before", [False, True])
def test_forward_with_long_rows_is_captured(listed_before):
    """Rows of 129 to 1,024 edges under a known bound: a forward recorded into a CUDA graph needs no host read, whether or not the
    graph's work list was made before."""
    from budgetformer_b200.ops.edge_attention import edge_attention, edge_attention_reference
    graph = _graph(700, 400, 21, False)
    graph.max_degree = 400
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (torch.randn(700, 4, 16, generator=gen, device="cuda") for _ in range(3))
    with torch.no_grad():
        edge_attention(q, k, v, _graph(700, 5, 1, False))                  # the kernels are loaded
        if listed_before:
            edge_attention(q, k, v, graph)
        torch.cuda.synchronize()
        rec = torch.cuda.CUDAGraph()
        with torch.cuda.graph(rec):
            out = edge_attention(q, k, v, graph)
        out.zero_()
        rec.replay()
        torch.cuda.synchronize()
    ref = edge_attention_reference(q, k, v, graph)
    assert float((out - ref).norm()) <= 2e-5 * float(ref.norm())


@pytest.mark.parametrize("n", [1, 33, 8192, 8193, 20011])
def test_work_lists_on_both_sides_of_the_sort(n):
    """The device's by-key view and work list against the CPU construction: keys of no, one, 64 and 65 edges and popular ones, below
    and above the number of keys from which single items are sorted by length; and the list of long query rows."""
    from budgetformer_b200.graph.attn_graph import LONG_CHUNK, LONG_ROW, AttnGraph
    gen = torch.Generator().manual_seed(n)
    src = (torch.rand(6 * n, generator=gen) ** 4 * n).long().clamp_(max=n - 1)
    src = torch.cat([src, torch.full((64,), n - 1), torch.full((65,), n // 2), torch.full((200,), n // 3)])
    dst = torch.cat([torch.randint(0, n, (6 * n,), generator=gen), torch.full((329,), n // 5)])
    ref = AttnGraph.from_edge_index(torch.stack([src, dst]), n).ensure_transpose()
    dev = AttnGraph(n, ref.rowptr.cuda(), ref.col.cuda()).ensure_transpose()
    for name in ("t_rowptr", "t_row", "t_eid", "t_task", "t_split"):
        assert torch.equal(getattr(ref, name), getattr(dev, name).cpu()), name
    assert ref.kv_slots == dev.kv_slots
    deg = (ref.rowptr[1:] - ref.rowptr[:-1]).tolist()
    tasks, splits = [], []
    for row, d in enumerate(deg):
        if d > LONG_ROW:
            items = [(row, int(ref.rowptr[row]) + c, int(ref.rowptr[row]) + min(c + LONG_CHUNK, d)) for c in range(0, d, LONG_CHUNK)]
            splits.append([row, len(tasks), len(items)])
            tasks += [[*it, len(tasks) + i] for i, it in enumerate(items)]
    task, split, least = dev.long_rows()
    assert task.tolist() == tasks and split.tolist() == splits and least == LONG_ROW


def test_backward_without_room_for_the_score_gradients():
    """The buffer of kept score gradients is the largest thing a backward pass allocates.  Where the allocator cannot give it, the
    scores are computed twice: the same gradients up to the order of fp32 sums."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    n, deg = 4000, 2000
    gen = torch.Generator(device="cuda").manual_seed(6)
    dst = torch.arange(n, device="cuda").repeat_interleave(deg)
    graph = AttnGraph.from_edge_index(torch.stack([torch.randint(0, n, (n * deg,), generator=gen, device="cuda"), dst]), n).ensure_transpose()
    graph.long_rows()
    del dst
    q, k, v, dout = (torch.randn(n, 8, 8, generator=gen, device="cuda") for _ in range(4))
    args = [t.requires_grad_() for t in (q, k, v)]
    want = torch.autograd.grad(edge_attention(*args, graph), args, dout)
    out = edge_attention(*args, graph)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (200 << 20)) / total)   # the buffer takes 256 MB
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got = torch.autograd.grad(out, args, dout)
        assert torch.cuda.max_memory_allocated() - before < n * deg * 8 * 4
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, want):
        assert float((a - b).norm()) <= 2e-5 * (float(b.norm()) + float(dout.norm()))


@pytest.mark.parametrize("n,heads,hn,dtype", [(257, 8, 16, torch.bfloat16), (240007, 8, 16, torch.bfloat16), (101021, 4, 64, torch.float32)])
def test_output_dropout_in_both_forward_kernels(n, heads, hn, dtype):
    """Dropout fused into the stored output, on the sizes of either kernel: the plain output where the hash keeps, scaled, else 0."""
    from budgetformer_b200.ops import _ext
    from budgetformer_b200.ops.gemm import hash_keep_mask
    graph = _graph(n, 3, 12, False)
    gen = torch.Generator(device="cuda").manual_seed(8)
    q, k, v = (torch.randn(n, heads, hn, generator=gen, device="cuda").to(dtype) for _ in range(3))
    res = []
    for drop in ([], [0.25, 9.0, float(n), 0.0]):
        out, z = torch.empty_like(q), torch.empty(n, heads, device="cuda")
        _ext.load().edge_attn_fwd(q, k, v, out, z, graph.rowptr, graph.col, None, None, 0, 0.0, 0, 3, drop, [])
        res.append((out.float().flatten(1), z))
    keep = hash_keep_mask(9, n, heads * hn, 0.25, "cuda")
    want = torch.where(keep, res[0][0] / 0.75, torch.zeros((), device="cuda"))
    unit = {torch.float32: 2.0 ** -20, torch.bfloat16: 2.0 ** -7}[dtype]        # both are rounded; fp32: another order of sums
    assert bool(((res[1][0] - want).abs() <= unit * want.abs() + 1e-6).all())
    assert float((res[0][1] - res[1][1]).norm()) <= 1e-6 * float(res[0][1].norm())


def test_by_key_view_without_its_work_list():
    """A graph that was given t_rowptr, t_row and t_eid alone: the backward pass makes the work list, and the gradients are those
    of the graph's own."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    whole = _graph(900, 60, 3, False).ensure_transpose()
    assert whole.kv_slots > 0
    part = AttnGraph(whole.num_rows, whole.rowptr, whole.col, None, whole.t_rowptr, whole.t_row, whole.t_eid)
    gen = torch.Generator(device="cuda").manual_seed(2)
    q, k, v, dout = (torch.randn(900, 4, 16, generator=gen, device="cuda") for _ in range(4))
    args = [t.requires_grad_() for t in (q, k, v)]
    for a, b in zip(*(torch.autograd.grad(edge_attention(*args, g), args, dout) for g in (whole, part))):
        assert torch.equal(a, b)


@pytest.mark.parametrize("heads,variant,dtype", [(40, "exphormer", torch.bfloat16), (48, "exphormer", torch.float32), (48, "plain", torch.bfloat16)])
def test_attention_of_wide_rows(heads, variant, dtype):
    """Rows of 5,120 and 6,144 elements with long queries and split keys: the type table's gradient and the sums of split rows
    need more shared memory than a block gets by default, or have to do without."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    gen = torch.Generator().manual_seed(heads)
    n, hn = 61, 128
    dst = torch.cat([torch.zeros(200, dtype=torch.long), torch.arange(n).repeat_interleave(4)])
    src = torch.randint(0, n, (dst.numel(),), generator=gen)
    src[200:300] = 7                                                       # a split key
    graph = AttnGraph.from_edge_index(torch.stack([src, dst, torch.randint(0, 2, (dst.numel(),), generator=gen)]), n).to("cuda")
    q, k, v, dout = (torch.randn(n, heads, hn, generator=gen).cuda().to(dtype) for _ in range(4))
    tab = torch.randn(2, heads, hn, generator=gen).cuda() if variant == "exphormer" else None
    want = _reference(q, k, v, dout, graph, tab, variant, 0.0, 0)
    args = [x.requires_grad_() for x in (q, k, v)] + ([tab.requires_grad_()] if tab is not None else [])
    out = edge_attention(q, k, v, graph, variant=variant, etable=tab)
    got = [out] + list(torch.autograd.grad(out, args, dout))
    tol = {torch.float32: 2e-5, torch.bfloat16: 2.5e-2}[dtype]             # as in test_attention_streams
    for a, b in zip(got, want):
        assert float((a.double() - b.double()).norm()) <= tol * (float(b.double().norm()) + float(dout.double().norm()))


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


@pytest.mark.parametrize("long_row", [False, True])
def test_typed_attention_keeps_the_other_type_finite(long_row):
    """A row of the type table that no edge carries, and an infinite key that only edges of one type name, leave the gradients of the
    other type as they are: nothing is multiplied by an absent type."""
    from budgetformer_b200.graph.attn_graph import AttnGraph
    from budgetformer_b200.ops.edge_attention import edge_attention
    n, deg = 301, 5
    dst = torch.arange(n).repeat_interleave(deg)
    if long_row:
        dst = torch.cat([torch.zeros(300, dtype=torch.long), dst])
    src = (torch.arange(dst.numel()) * 7 + 3) % n
    typ = (dst % 2 == 1).long()                                            # odd queries: type 1 alone
    src[src == 9] = 10
    src[dst == 51] = 9                                                     # only query 51 (type 1) names key 9
    graph = AttnGraph.from_edge_index(torch.stack([src, dst, typ]), n).to("cuda")
    q, k, v, dout = (torch.randn(n, 4, 16, device="cuda") for _ in range(4))
    k[9] = float("inf")
    tab = torch.randn(2, 4, 16, device="cuda")
    args = [t.requires_grad_() for t in (q, k, v, tab)]
    grads = torch.autograd.grad(edge_attention(q, k, v, graph, variant="exphormer", etable=tab), args, dout)
    assert torch.isfinite(grads[3][0]).all() and torch.isfinite(grads[0][::2]).all()
    with torch.no_grad():
        k[9] = 0.0
        tab[1] = float("inf")
    grads = torch.autograd.grad(edge_attention(q, k, v, graph, variant="exphormer", etable=tab), args, dout)
    assert torch.isfinite(grads[0][::2]).all() and torch.isfinite(grads[3][0]).all()
    even = torch.ones(n, dtype=torch.bool, device="cuda")
    even[src[typ == 1].cuda()] = False                                     # keys that no edge of type 1 names
    assert even.any() and torch.isfinite(grads[1][even]).all()


@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 1, 0), (63, 64, 64, 0), (65, 60, 68, 0), (1000, 47, 101, 0), (4097, 256, 64, 4),
                                       (20011, 64, 256, 0), (300, 130, 70, 1)])
def test_f32_weight_grad(m, n, k, pad):
    from budgetformer_b200.ops import _ext
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    dy = torch.randn(m, n + pad, generator=gen, device="cuda")[:, :n]
    x = torch.randn(m, k + pad, generator=gen, device="cuda")[:, :k]
    for bias in (True, False):
        flat = _ext.load().f32_weight_grad(dy, x, bias)
        want, size = dy.double().t() @ x.double(), dy.double().abs().t() @ x.double().abs()
        # any order of m products and additions: |error| <= m * 2^-24 * sum |dy| |x|
        assert bool(((flat[:n * k].view(n, k).double() - want).abs() <= m * 2.0 ** -24 * size + 1e-30).all())
        if bias:
            db = dy.double().sum(0)
            assert bool(((flat[n * k:].double() - db).abs() <= m * 2.0 ** -24 * dy.double().abs().sum(0) + 1e-30).all())


@pytest.mark.parametrize("out_features,in_features", [(1, 24), (24, 1), (1, 1)])
@pytest.mark.parametrize("rows", [128, 1003])
def test_fp32_linear_of_one_column(out_features, in_features, rows):
    """One output or one feature whose matrix is a transposed row: its column stride is not 1 and means nothing."""
    from budgetformer_b200.ops.gemm import linear_f32
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(in_features, rows, generator=gen, device="cuda").t() if in_features == 1 else torch.randn(rows, in_features, device="cuda")
    w = torch.randn(out_features, in_features, generator=gen, device="cuda", requires_grad=True)
    b = torch.randn(out_features, generator=gen, device="cuda", requires_grad=True)
    probe = torch.randn(out_features, rows, generator=gen, device="cuda")
    for loss in (lambda y: (y.t() * probe).sum(), lambda y: torch.softmax(y.t(), 1).pow(2).sum(), lambda y: y.sum()):
        got = torch.autograd.grad(loss(linear_f32(x, w, b)), (w, b))
        wd, bd = w.detach().double().requires_grad_(), b.detach().double().requires_grad_()
        y = torch.nn.functional.linear(x.double(), wd, bd)
        want = torch.autograd.grad(loss(y), (wd, bd))
        for u, v in zip(got, want):
            # sums of `rows` products of values of order 1 in any order, and fp32 rounding of dy itself
            assert u.shape == v.shape and float((u.double() - v).abs().max()) <= rows * 2.0 ** -23


@pytest.mark.parametrize("out_features,in_features", [(0, 8), (8, 0), (0, 0)])
def test_fp32_linear_of_no_width(out_features, in_features):
    """No outputs or no features: zeros and empty tensors, as PyTorch's linear layer gives."""
    from budgetformer_b200.ops.gemm import linear_f32
    x = torch.randn(300, in_features, device="cuda", requires_grad=True)
    w = torch.randn(out_features, in_features, device="cuda", requires_grad=True)
    b = torch.randn(out_features, device="cuda", requires_grad=True)
    res = []
    for f in (linear_f32, torch.nn.functional.linear):
        y = f(x, w, b)
        res.append([y] + list(torch.autograd.grad(y.sum(), (x, w, b))))
    for u, v in zip(*res):
        assert u.shape == v.shape and torch.equal(u, v)


def test_fp32_linear_leaves_wide_layers_and_tf32_to_the_library(monkeypatch):
    from budgetformer_b200.ops import gemm
    calls = []
    monkeypatch.setattr(gemm._LinearF32, "apply", lambda *a: calls.append(1) or torch.nn.functional.linear(*a))
    for rows, n, k, kernel in ((4096, 64, 64, True), (4096, 512, 512, False), (9000, 64, 1433, False), (9000, 1, 256, False), (300, 1, 256, True)):
        x, w = torch.randn(rows, k, device="cuda"), torch.randn(n, k, device="cuda", requires_grad=True)
        calls.clear()
        gemm.linear_f32(x, w)
        assert bool(calls) == kernel, (rows, n, k)
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", True)
    calls.clear()
    gemm.linear_f32(torch.randn(4096, 64, device="cuda"), torch.randn(64, 64, device="cuda", requires_grad=True))
    assert not calls


def test_fp32_modules_match_torch():
    """The models' call of a linear layer and the row-kernel LayerNorm against torch's, first and second derivative, few and many
    rows."""
    from budgetformer_b200.models.common import linear
    from budgetformer_b200.ops.norm import layer_norm

    class Linear(torch.nn.Module):
        def __init__(self, k, n):
            super().__init__()
            self.weight, self.bias = (torch.nn.Parameter(torch.randn(*size) * k ** -0.5) for size in ((n, k), (n,)))

        def forward(self, x):
            inner = torch.nn.Linear(self.weight.size(1), self.weight.size(0), device="meta")
            inner.weight, inner.bias = self.weight, self.bias
            return linear(inner, x)

    class LayerNorm(torch.nn.LayerNorm):
        def forward(self, x):
            return layer_norm(x[0], self.weight, self.bias, self.eps)[None]

    for rows in (7, 3000):
        for cls, ref, args in ((Linear, torch.nn.Linear, (24, 40)), (LayerNorm, torch.nn.LayerNorm, (24,))):
            torch.manual_seed(rows)
            a, b = cls(*args).cuda(), ref(*args).cuda()
            b.load_state_dict(a.state_dict())
            x = torch.randn(1, rows, 24, device="cuda")
            res = []
            weights = torch.randn_like(a(x)).detach()                      # sum(y^2) alone is constant behind a LayerNorm
            for mod in (a, b):
                xi = x.clone().requires_grad_()
                y = mod(xi)
                g1 = torch.autograd.grad((y * y * weights).sum(), [xi] + list(mod.parameters()), retain_graph=True)
                g2 = torch.autograd.grad((y * y * y * weights).sum(), xi, create_graph=True)[0]
                g2 = torch.autograd.grad((g2 * g2).sum(), [xi] + list(mod.parameters()), allow_unused=True)
                res.append([y] + list(g1) + [g for g in g2 if g is not None])
            assert len(res[0]) == len(res[1])
            for u, w in zip(*res):
                assert float((u - w).norm()) <= 2e-5 * float(w.norm()) + 1e-6


@pytest.mark.parametrize("rows,cols,dtype", [(1, 8, torch.bfloat16), (37, 24, torch.float16), (4099, 256, torch.bfloat16),
                                             (515, 2048, torch.bfloat16), (700, 136, torch.float32)])
def test_row_element_kernels(rows, cols, dtype):
    """BatchNorm's affine passes and the hashed dropout: fp32 arithmetic, one rounding."""
    from budgetformer_b200.ops import _ext
    from budgetformer_b200.ops.gemm import hash_keep_mask
    from budgetformer_b200.ops.norm import gelu_dropout, hash_dropout
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, cols + 8, generator=gen, device="cuda").to(dtype)[:, :cols]      # row pitch wider than the row
    z = torch.randn(rows, cols, generator=gen, device="cuda").to(dtype)
    a, b, c = (torch.randn(cols, generator=gen, device="cuda") for _ in range(3))
    unit = {torch.float32: 2.0 ** -23, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[dtype]
    ext = _ext.load()
    for got, want, size in ((ext.col_affine(x, None, a, b, None), x.double() * a + b, (x.double() * a).abs() + b.abs()),
                            (ext.col_affine(x, z, a, b, c), z.double() * a + x.double() * b + c,
                             (z.double() * a).abs() + (x.double() * b).abs() + c.abs())):
        assert bool(((got.double() - want).abs() <= unit * size + 1e-7).all())
    keep = hash_keep_mask(5, rows, cols, 0.25, "cuda")
    want = torch.where(keep, x.float() * (1.0 / 0.75), torch.zeros((), device="cuda"))
    assert bool(((hash_dropout(x, 5, 0.25).float() - want).abs() <= unit * want.abs() + 1e-7).all())
    want = torch.where(keep, torch.nn.functional.gelu(x.float()) * (1.0 / 0.75), torch.zeros((), device="cuda"))
    assert bool(((gelu_dropout(x, 5, 0.25).float() - want).abs() <= unit * want.abs() + 1e-6).all())


def test_type_table_at_any_address():
    """Tables that are views at odd offsets give what an aligned copy gives, forward and backward; so does one row for a list of one type."""
    from budgetformer_b200.ops.edge_attention import edge_attention
    from helpers import random_attn_graph
    graph = random_attn_graph(typed=True).to("cuda")
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, dout = (torch.randn(graph.rowptr.numel() - 1, 4, 16, generator=g, device="cuda").bfloat16() for _ in range(4))
    flat = torch.randn(2 * 64 + 4, generator=g, device="cuda")

    def grads(table):
        args = [t.detach().requires_grad_() for t in (q, k, v, table)]
        out = edge_attention(*args[:3], graph, variant="exphormer", etable=args[3])
        return [out] + list(torch.autograd.grad(out, args, dout))

    for off in (1, 2, 3):
        view = flat[off:off + 128].view(2, 4, 16)
        assert view.data_ptr() % 16
        for x, y in zip(grads(view), grads(view.clone())):
            assert torch.allclose(x.float(), y.float(), rtol=1e-5, atol=1e-5)     # the table's gradient meets in atomics
    graph.etype.zero_()
    table = flat[:128].view(2, 4, 16).clone()
    one, two = grads(table[:1]), grads(table)
    for x, y in zip(one[:4], two[:4]):
        assert torch.equal(x, y)
    assert torch.allclose(one[4], two[4][:1], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("heads,hn,dtype", [(9, 128, torch.bfloat16), (4, 64, torch.float32), (3, 8, torch.float16), (8, 16, torch.bfloat16)])
@pytest.mark.parametrize("variant", ["plain", "gps"])
def test_an_absent_edge_is_not_multiplied(heads, hn, dtype, variant):
    """Rows and keys of odd length are padded to pairs by some of the kernels: an infinity in the last edge's value or output gradient
    comes out as one, not as the NaN that weight 0 makes of it."""
    from budgetformer_b200.ops.edge_attention import edge_attention
    n, gen = 700, torch.Generator().manual_seed(hn)
    deg = torch.arange(n) % 8
    dst = torch.repeat_interleave(torch.arange(n), deg)
    graph = _graph_of(torch.stack([torch.randint(0, n, (dst.numel(),), generator=gen), dst]), n)
    gen = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v, dout = (torch.randn(n, heads, hn, generator=gen, device="cuda").to(dtype) for _ in range(4))
    bad = torch.zeros(n, heads, hn, dtype=torch.bool, device="cuda")
    bad.view(-1)[torch.randint(0, bad.numel(), (40,), generator=gen, device="cuda")] = True
    neg = v.masked_fill(bad, float("-inf"))
    out = edge_attention(q, k, neg, graph, variant=variant)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), graph.rowptr.diff().long())
    hit = torch.zeros(n, heads, hn, dtype=torch.int32, device="cuda").index_add_(0, rows, bad[graph.col.long()].int()) > 0
    assert hit.any() and torch.equal(out == float("-inf"), hit) and not out.isnan().any()
    args = [x.detach().requires_grad_() for x in (q, k, v)]
    grads = torch.autograd.grad(edge_attention(*args, graph, variant=variant), args, dout.masked_fill(bad, float("inf")))
    hit = torch.zeros(n, heads, hn, dtype=torch.int32, device="cuda").index_add_(0, graph.col.long(), bad[rows].int()) > 0
    assert hit.any() and torch.equal(grads[2] == float("inf"), hit) and not grads[2].isnan().any()

