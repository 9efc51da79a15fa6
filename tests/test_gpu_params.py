"""Weight copies and gradient buckets (csrc/param_kernels.cu) against PyTorch's operators."""
import pytest
import torch

from budgetformer_b200.ops import gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n,k", [(1, 1), (31, 33), (128, 269), (96, 64)])
def test_operand_copies_follow_their_weights(n, k, dtype):
    """Copies equal the cast weight, as it is and transposed; a change of one weight renews every copy in use, and a copy that someone
    still holds keeps its values."""
    torch.manual_seed(n + k)
    ws = [torch.nn.Parameter(torch.randn(n, k, device="cuda")) for _ in range(70)]      # more than one launch's table
    for step in range(3):
        held = gemm.operand_copy(ws[0], dtype)
        before = held.clone()
        for w in ws:
            assert torch.equal(gemm.operand_copy(w, dtype), w.detach().to(dtype))
            assert torch.equal(gemm.operand_copy(w, dtype, transpose=True), w.detach().to(dtype).t())
        with torch.no_grad():
            for w in ws:
                w.add_(1.0 + step)
        fresh = gemm.operand_copy(ws[0], dtype)
        assert fresh is not held and torch.equal(held, before) and torch.equal(fresh, ws[0].detach().to(dtype))
    with torch.no_grad():
        ws[3].data.mul_(2.0)                                # the storage, past the version counter, as a flat optimizer does
    gemm.weights_changed()
    assert torch.equal(gemm.operand_copy(ws[3], dtype), ws[3].detach().to(dtype))


def test_operand_copies_of_another_stream_are_left_alone():
    """A copy that was last used on another stream is not rebuilt by this one: nothing would order the two."""
    a, b = (torch.nn.Parameter(torch.randn(64, 64, device="cuda")) for _ in range(2))
    side = torch.cuda.Stream()
    gemm.operand_copy(a, torch.bfloat16)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        on_side = gemm.operand_copy(b, torch.bfloat16)
    gemm.weights_changed()
    gemm.operand_copy(a, torch.bfloat16)
    recipe = gemm._RECIPES[(id(b), torch.bfloat16, False, "")]
    assert recipe.out is on_side
    torch.cuda.synchronize()


def test_operand_copies_follow_their_own_optimizer():
    """A step of one optimizer leaves the copies of another's weights as they are."""
    a, b, c = (torch.nn.Parameter(torch.randn(16, 24, device="cuda")) for _ in range(3))
    first, second = [0], [0]
    gemm.watch_weights([a, b], first)
    gemm.watch_weights([c], second)
    copy = lambda p: gemm.operand_copy(p, torch.bfloat16)
    before = [copy(p) for p in (a, b, c)]
    with torch.no_grad():
        a.data.add_(1.0)
        b.data.add_(1.0)
    gemm.weights_changed(first)
    assert torch.equal(copy(a), a.detach().bfloat16()) and copy(a) is not before[0]
    recipe = gemm._RECIPES[(id(b), torch.bfloat16, False, "")]
    assert recipe.out is not before[1] and torch.equal(copy(b), b.detach().bfloat16())      # made along with a's
    assert copy(c) is before[2]


def test_a_copy_made_on_one_stream_is_ready_on_another():
    """A stream that finds a copy which another one made waits for its launch; from then on the maker's stream no longer renews it along
    with others, since nothing would order the two."""
    a, b = (torch.nn.Parameter(torch.randn(256, 256, device="cuda")) for _ in range(2))
    counter = [0]
    gemm.watch_weights([a, b], counter)
    side = torch.cuda.Stream()
    for p in (a, b):
        gemm.operand_copy(p, torch.bfloat16)
    recipe = gemm._RECIPES[(id(b), torch.bfloat16, False, "")]
    for step in range(2):
        before = recipe.out
        torch.cuda._sleep(100_000_000)                       # some 50 ms: the copies' launch lies behind it
        with torch.no_grad():
            a.data.add_(1.0)
            b.data.add_(1.0)
        gemm.weights_changed(counter)
        gemm.operand_copy(a, torch.bfloat16)
        assert (recipe.out is before) == (step == 1)         # renewed by the main stream the first time only
        with torch.cuda.stream(side):
            got = gemm.operand_copy(b, torch.bfloat16).clone()
        side.synchronize()
        if step == 0:
            assert torch.equal(got, b.detach().bfloat16())
    torch.cuda.synchronize()


def test_only_what_the_announced_step_made_stale_is_renewed_along():
    """Copies of weights that no watched optimizer owns, or that were written again after its step, wait for their own request: the
    stream that renews another copy does not know when they are written."""
    a, b, c, d = (torch.nn.Parameter(torch.randn(32, 32, device="cuda")) for _ in range(4))
    recipe = lambda p: gemm._RECIPES[(id(p), torch.bfloat16, False, "")]
    copy = lambda p: gemm.operand_copy(p, torch.bfloat16)
    opt = torch.optim.SGD([a, b, c], lr=0.5)
    gemm.watch_optimizer(opt)
    before = [copy(p) for p in (a, b, c, d)]
    for p in (a, b, c):
        p.grad = torch.ones_like(p)
    opt.step()
    with torch.no_grad():
        c.add_(1.0)
        d.add_(1.0)
    assert torch.equal(copy(a), a.detach().bfloat16())
    assert recipe(b).out is not before[1] and recipe(c).out is before[2] and recipe(d).out is before[3]
    for p in (b, c, d):
        assert torch.equal(copy(p), p.detach().bfloat16())


def test_a_copy_of_a_recorded_launch_is_not_found_by_others():
    """A forward pass that is recorded before any other makes its copies inside the graph: an eager pass before the first replay makes
    its own."""
    from budgetformer_b200.ops.gemm import fused_linear
    lin = torch.nn.Linear(64, 32).cuda()
    x = torch.randn(128, 64, device="cuda").bfloat16()
    other = torch.nn.Linear(64, 32).cuda()
    torch.cuda.synchronize()
    with torch.no_grad():
        fused_linear(x, other.weight, other.bias)            # the launch's own first use is no part of this
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = fused_linear(x, lin.weight, lin.bias)
        eager = fused_linear(x, lin.weight, lin.bias)
        want = torch.nn.functional.linear(x.float(), lin.weight.bfloat16().float(), lin.bias)
        assert torch.allclose(eager.float(), want, rtol=2.0 ** -7, atol=2.0 ** -7)
        graph.replay()
        assert torch.equal(out, eager)


def _net():
    torch.manual_seed(2)
    return torch.nn.Sequential(torch.nn.Linear(37, 65), torch.nn.ReLU(), torch.nn.Linear(65, 3, bias=False), torch.nn.Linear(3, 1)).cuda()


def test_gradient_bucket_gathers_what_the_backward_pass_left():
    """Gradients equal PyTorch's; one without a gradient is zero; several backward passes add up; the bucket is complete whether it is
    read after ``finalize_backward`` or before; and ``param.grad`` is a view of it afterwards."""
    from budgetformer_b200.parallel.reducer import GradientReducer
    net, ref = _net(), _net()
    unused = torch.nn.Parameter(torch.ones(5, 7, device="cuda"))
    net.register_parameter("unused", unused)
    red = GradientReducer(net, None, 25.0, 1)
    x = torch.randn(50, 37, device="cuda")
    for passes, finalize in ((1, True), (2, True), (1, False), (0, True)):
        red.prepare_backward()
        ref.zero_grad()
        for _ in range(passes):
            net(x).square().mean().backward()
            ref(x).square().mean().backward()
        if finalize:
            red.finalize_backward()
        flat = torch.cat([b.flat for b in red.buckets])
        for p, q in zip(list(net.parameters())[1:], ref.parameters()):
            want = torch.zeros_like(q) if q.grad is None else q.grad
            assert torch.equal(p.grad, want)
        assert not unused.grad.any()
        for b in red.buckets:
            for p, off in zip(b.params, b.offsets):
                assert p.grad.data_ptr() == b.flat.data_ptr() + 4 * off
        assert float(flat.abs().sum()) > 0 or passes == 0


def test_gradient_bucket_takes_any_gradient():
    """Expanded, transposed, sparse and in-place gradients that a program puts on a parameter land in the bucket."""
    from budgetformer_b200.parallel.reducer import GradientReducer
    m = torch.nn.ParameterList([torch.nn.Parameter(torch.randn(6, 9, device="cuda")) for _ in range(4)])
    red = GradientReducer(m, None, 25.0, 1)
    red.prepare_backward()
    t = torch.randn(9, 6, device="cuda")
    m[0].grad = torch.randn(9, device="cuda").expand(6, 9)
    m[1].grad = t.t()
    m[2].grad = torch.randn(6, 9, device="cuda").to_sparse()
    want = [m[0].grad.clone(), t.t().clone(), m[2].grad.to_dense(), torch.zeros(6, 9, device="cuda")]
    red.finalize_backward()
    for p, w in zip(m, want):
        assert torch.equal(p.grad, w) and p.grad.is_contiguous()


def test_gradient_bucket_read_on_a_side_stream():
    """Whoever reads the bucket first gathers the gradients, on its own stream: the training loop's stream, and a third one that reads it
    afterwards, see them complete."""
    from budgetformer_b200.parallel.reducer import GradientReducer
    net, ref = _net(), _net()
    red = GradientReducer(net, None, 25.0, 1)
    x = torch.randn(50, 37, device="cuda")
    main, side, third = torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(2):
        ref.zero_grad()
        ref(x).square().mean().backward()
        red.prepare_backward()
        net(x).square().mean().backward()
        done = main.record_event()
        side.wait_event(done)
        third.wait_event(done)
        with torch.cuda.stream(side):
            torch.cuda._sleep(50_000_000)                    # some 25 ms in front of the gather
            on_side = [b.flat.clone() for b in red.buckets]
        on_main = [p.grad.clone() for p in net.parameters()]
        with torch.cuda.stream(third):
            on_third = [b.flat.clone() for b in red.buckets]
        torch.cuda.synchronize()
        for got, q in zip(on_main, ref.parameters()):
            assert torch.equal(got, q.grad)
        for a, b in zip(on_side, on_third):
            assert torch.equal(a, b)
        with torch.no_grad():
            for p, q in zip(net.parameters(), ref.parameters()):
                p.mul_(1.25)
                q.mul_(1.25)
