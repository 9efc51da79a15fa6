"""tcgen05 GEMM against fp32 PyTorch matmul of the same operands."""
import pytest
import torch

from budgetformer_b200.ops import gemm

pytestmark = pytest.mark.gpu


def _ref(a, w, bias=None, act=None, residual=None, mask=None, drop=None, scale=1.0):
    y = a.float() @ w.float().t() * scale
    if bias is not None:
        y = y + bias.float()
    if act == "relu":
        y = torch.relu(y)
    elif act == "gelu":
        y = torch.nn.functional.gelu(y)
    if drop is not None:
        p, seed = drop
        keep = gemm.hash_keep_mask(seed, y.size(0), y.size(1), p, y.device)
        y = torch.where(keep, y / (1 - p), torch.zeros_like(y))
    if mask is not None:
        y = torch.where(mask.float() > 0, y, torch.zeros_like(y))
    if residual is not None:
        y = y + residual.float()
    return y


def _close(got, want, dtype):
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    scale = max(1.0, float(want.abs().max()))
    err = float((got.float() - want).abs().max())
    assert err <= tol * scale, f"max err {err} scale {scale}"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k", [(128, 128, 128), (1000, 384, 128), (333, 256, 256), (4096, 768, 256),
                                   (129, 64, 64), (70000, 128, 256), (257, 192, 512), (64, 16, 64), (5000, 48, 128),
                                   (3000, 64, 32), (3000, 32, 16), (777, 128, 40)])
def test_gemm_plain(m, n, k, dtype):
    torch.manual_seed(0)
    a = torch.randn(m, k, device="cuda").to(dtype)
    w = (torch.randn(n, k, device="cuda") / k ** 0.5).to(dtype)
    out = gemm.gemm_tn(a, w)
    gemm.check_status("cuda")
    _close(out, _ref(a, w), dtype)


def test_gemm_fp32_output_and_scale():
    a = torch.randn(500, 128, device="cuda").bfloat16()
    w = torch.randn(128, 128, device="cuda").bfloat16() * 0.1
    out = gemm.gemm_tn(a, w, out_scale=0.5, out_dtype=torch.float32)
    gemm.check_status("cuda")
    assert out.dtype == torch.float32
    assert torch.allclose(out, _ref(a, w, scale=0.5), atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("act", [None, "relu", "gelu"])
def test_gemm_epilogues(act):
    torch.manual_seed(1)
    m, n, k = 3000, 256, 128
    a = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.1).bfloat16()
    bias = torch.randn(n, device="cuda")
    res = torch.randn(m, n, device="cuda").bfloat16()
    out = gemm.gemm_tn(a, w, bias, act, residual=res)
    _close(out, _ref(a, w, bias, act, res), torch.bfloat16)
    out = gemm.gemm_tn(a, w, bias, act, dropout_p=0.3, dropout_seed=77)
    _close(out, _ref(a, w, bias, act, drop=(0.3, 77)), torch.bfloat16)
    mask = torch.randn(m, n, device="cuda").bfloat16()
    out = gemm.gemm_tn(a, w, relu_mask=mask)
    _close(out, _ref(a, w, mask=mask), torch.bfloat16)
    gemm.check_status("cuda")


# One panel and several, groups of panels in one and in several chunks, column groups on different blocks, weights that stay in shared
# memory and weights that stream; ragged rows (a warp without any, one row), panels cut by N, K with a zero-filled tail.
_ROW_SHAPES = [(1, 64, 64), (31, 16, 16), (33, 48, 72), (128, 128, 128), (129, 384, 128), (8191, 192, 64), (4097, 80, 272),
               (2500, 320, 128), (2049, 448, 64), (40001, 128, 384), (30011, 768, 256), (20003, 256, 512), (19001, 256, 768),
               (1500, 512, 1024), (60000, 1024, 256)]
_ROW_EPILOGUES = ["none", "bias", "drop", "res", "bias drop", "bias res", "bias drop res", "bias relu", "bias gelu", "bias relu bits",
                  "bias relu drop bits", "mask", "mask scale", "gelugrad", "gelugrad drop", "bias gelu z", "bias gelu drop z"]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k", _ROW_SHAPES)
def test_gemm_row_streaming_epilogues(m, n, k, dtype):
    """Every epilogue against fp32 products, into a view of a larger matrix whose other elements stay as they are.  One rounding to 16
    bits (half a unit in the last of 8 or 11 places: 2^-8, 2^-11 of the value), the operands' products added up in fp32, and 2^-20 for the activations."""
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").to(dtype)
    w = (torch.randn(n, k, device="cuda") / k ** 0.5).to(dtype)
    bias = torch.randn(n, device="cuda")
    side = torch.randn(m, n, device="cuda").to(dtype)
    base = a.double() @ w.double().t()
    slack = (a.double().abs() @ w.double().abs().t() + 4) * k ** 0.5 * 2.0 ** -22 + 2.0 ** -20
    p, seed = 0.3125, 77                                 # a float: the kernel takes its threshold from one
    keep = gemm.hash_keep_mask(seed, m, n, p, "cuda")
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    bits = torch.randint(-2 ** 15, 2 ** 15, (n // 16, m), device="cuda").to(torch.int16)
    unpack = lambda b: torch.stack([(b.int() >> i) & 1 for i in range(16)], 1).reshape(n, m).t().bool()
    for epi in _ROW_EPILOGUES:
        f = epi.split()
        kw, want = {}, base.clone()
        big = torch.full((m + 2, n + 8), 7.0, device="cuda", dtype=dtype)
        out = big[1:m + 1, :n]
        if "scale" in f:
            kw["out_scale"] = 1.25
            want = want * 1.25
        if "bias" in f:
            want = want + bias.double()
        z = None
        if "z" in f:
            z = kw["z_out"] = torch.empty(m, n, device="cuda", dtype=dtype)
        if "relu" in f:
            kw["act"] = "relu"
            want = want.clamp(min=0)
        if "gelu" in f:
            kw["act"] = "gelu"
        if "mask" in f:
            kw["relu_bits_in"] = bits
        if "bits" in f:
            kw["relu_bits_out"] = torch.zeros_like(bits)
        if "res" in f:
            kw["residual"] = side
        if "gelugrad" in f:
            kw["gelu_grad_of"] = side
        if "drop" in f:
            kw.update(dropout_p=p, dropout_seed=seed)
        gemm.gemm_tn(a, w, bias if "bias" in f else None, out=out, **kw)
        gemm.check_status("cuda")
        if z is not None:
            assert ((z.double() - want).abs() <= slack + half_ulp * want.abs()).all(), epi
            want = z.double()
        if "gelu" in f:
            want = torch.nn.functional.gelu(want)
        if "drop" in f:
            want = torch.where(keep, want / (1 - p), 0.0)
        if "mask" in f:
            want = torch.where(unpack(bits), want, 0.0)
        if "gelugrad" in f:
            x = side.double()
            want = want * (0.5 * (1 + torch.erf(x / 2 ** 0.5)) + x * torch.exp(-x * x / 2) / (2 * torch.pi) ** 0.5)
        if "res" in f:
            want = want + side.double()
        err = (out.double() - want).abs() - (2 * slack + half_ulp * want.abs() * (1 + 2.0 ** -7))
        if dtype == torch.float16:
            err -= 2.0 ** -25                            # half a unit of the subnormals
        assert float(err.max()) <= 0, (epi, float(err.max()))
        if "bits" in f:
            got = unpack(kw["relu_bits_out"])
            assert torch.equal(got | (want.abs() < 4 * slack), (want > 0) | (want.abs() < 4 * slack)), epi
        edge = big.clone()
        edge[1:m + 1, :n] = 7.0
        assert bool((edge == 7.0).all()), epi


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,k", [(256, 256), (128, 384), (256, 512), (128, 128), (112, 264)])
def test_plain_products_of_many_rows(n, k, dtype):
    """Products with no epilogue but a bias around the number of rows (592 tiles) from which bf16 goes to either kernel by its shape."""
    torch.manual_seed(n + k)
    w = (torch.randn(n, k, device="cuda") / k ** 0.5).to(dtype)
    bias = torch.randn(n, device="cuda")
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for m in (591 * 128, 591 * 128 + 1, 592 * 128 + 37):
        a = torch.randn(m, k, device="cuda").to(dtype)
        base = a.double() @ w.double().t()
        for b in (None, bias):
            want = base if b is None else base + b.double()
            big = torch.full((m + 2, n + 8), 7.0, device="cuda", dtype=dtype)
            gemm.gemm_tn(a, w, b, out=big[1:m + 1, :n])
            gemm.check_status("cuda")
            # one rounding, and the products added up in fp32 (|a| |w| summed: about 0.64 k^0.5, at most 15, and the bias)
            err = (big[1:m + 1, :n].double() - want).abs() - half_ulp * want.abs() - 24 * k ** 0.5 * 2.0 ** -22
            assert float(err.max()) <= (2.0 ** -25 if dtype == torch.float16 else 0.0)
            assert bool((big[0] == 7.0).all()) and bool((big[m + 1] == 7.0).all()) and bool((big[:, n:] == 7.0).all())


def test_gemm_strided_input_rows():
    big = torch.randn(700, 3 * 128, device="cuda").bfloat16()
    a = big[:, 128:256]
    w = (torch.randn(64, 128, device="cuda") * 0.1).bfloat16()
    _close(gemm.gemm_tn(a, w), _ref(a, w), torch.bfloat16)


def test_fused_linear_autograd():
    torch.manual_seed(2)
    x = torch.randn(1500, 128, device="cuda").bfloat16().requires_grad_(True)
    lin = torch.nn.Linear(128, 256).cuda()
    res = torch.randn(1500, 256, device="cuda").bfloat16().requires_grad_(True)
    y = gemm.fused_linear(x, lin.weight, lin.bias, res, dropout_p=0.25, dropout_seed=5)
    dy = torch.randn_like(y)
    y.backward(dy)
    x2 = x.detach().float().requires_grad_(True)
    r2 = res.detach().float().requires_grad_(True)
    w2 = lin.weight.detach().bfloat16().float().requires_grad_(True)
    b2 = lin.bias.detach().clone().requires_grad_(True)
    keep = gemm.hash_keep_mask(5, 1500, 256, 0.25, "cuda")
    y2 = torch.where(keep, (x2 @ w2.t() + b2) / 0.75, torch.zeros(1, device="cuda")) + r2
    y2.backward(dy.float())
    _close(y.detach(), y2.detach(), torch.bfloat16)
    _close(x.grad, x2.grad, torch.bfloat16)
    _close(res.grad, r2.grad, torch.bfloat16)
    assert torch.allclose(lin.weight.grad, w2.grad, atol=0.03 * float(w2.grad.abs().max()), rtol=5e-2)
    assert torch.allclose(lin.bias.grad, b2.grad, atol=0.03 * float(b2.grad.abs().max()), rtol=5e-2)


@pytest.mark.parametrize("onchip_train", [False, True])
def test_fused_ffn_autograd(onchip_train, monkeypatch):
    from budgetformer_b200.ops import ffn as ffn_mod
    from budgetformer_b200.ops.ffn import fused_ffn
    from budgetformer_b200.ops import norm as bnorm
    # True: the training forward runs on the one-kernel form with the hidden matrix and the ReLU bits as side outputs
    monkeypatch.setattr(ffn_mod, "ONCHIP_FFN_TRAIN", onchip_train)
    torch.manual_seed(3)
    m, h = 2000, 128
    x = torch.randn(m, h, device="cuda").bfloat16().requires_grad_(True)
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    torch.manual_seed(11)
    y = fused_ffn(x, l1.weight, l1.bias, l2.weight, l2.bias, act="relu", residual=x, p1=0.2, p2=0.1, training=True)
    dy = torch.randn_like(y)
    y.backward(dy)
    torch.manual_seed(11)
    s1, s2 = bnorm.new_seed(), bnorm.new_seed()
    x2 = x.detach().float().requires_grad_(True)
    w1 = l1.weight.detach().bfloat16().float().requires_grad_(True)
    w2 = l2.weight.detach().bfloat16().float().requires_grad_(True)
    hdn = torch.relu(x2 @ w1.t() + l1.bias.detach())
    hdn = torch.where(gemm.hash_keep_mask(s1, m, 2 * h, 0.2, "cuda"), hdn / 0.8, torch.zeros(1, device="cuda"))
    hdn = hdn.bfloat16().float()
    o = hdn @ w2.t() + l2.bias.detach()
    o = torch.where(gemm.hash_keep_mask(s2, m, h, 0.1, "cuda"), o / 0.9, torch.zeros(1, device="cuda")) + x2
    o.backward(dy.float())
    _close(y.detach(), o.detach(), torch.bfloat16)
    _close(x.grad, x2.grad, torch.bfloat16)
    assert torch.allclose(l1.weight.grad, w1.grad, atol=0.03 * float(w1.grad.abs().max()), rtol=5e-2)
    assert torch.allclose(l2.weight.grad, w2.grad, atol=0.03 * float(w2.grad.abs().max()), rtol=5e-2)
    gemm.check_status("cuda")


@pytest.mark.parametrize("p1,p2", [(0.0, 0.0), (0.2, 0.1)])
def test_fused_gelu_ffn_autograd(p1, p2):
    """GELU feed-forward block (Graphormer): one pass gelu + dropout forward, and a backward whose hidden gradient
    (dropout mask regenerated, times gelu'(z)) comes out of the GEMM epilogue - against a float32 restatement with the
    same masks, rounded to bf16 where the fused path stores bf16."""
    from budgetformer_b200.ops.ffn import fused_ffn
    from budgetformer_b200.ops import norm as bnorm
    torch.manual_seed(5)
    m, h = 2500, 128
    x = torch.randn(m, h, device="cuda").bfloat16().requires_grad_(True)
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    torch.manual_seed(17)
    y = fused_ffn(x, l1.weight, l1.bias, l2.weight, l2.bias, act="gelu", residual=x, p1=p1, p2=p2, training=True)
    dy = torch.randn_like(y)
    y.backward(dy)
    gemm.check_status("cuda")
    torch.manual_seed(17)
    s1 = bnorm.new_seed() if p1 > 0 else 0
    s2 = bnorm.new_seed() if p2 > 0 else 0
    x2 = x.detach().float().requires_grad_(True)
    w1 = l1.weight.detach().bfloat16().float().requires_grad_(True)
    w2 = l2.weight.detach().bfloat16().float().requires_grad_(True)
    b1, b2 = l1.bias.detach().clone().requires_grad_(True), l2.bias.detach().clone().requires_grad_(True)
    z = x2 @ w1.t() + b1
    z = z + (z.bfloat16().float() - z).detach()                     # the fused path stores z in bf16
    hdn = torch.nn.functional.gelu(z)
    if p1 > 0:
        hdn = torch.where(gemm.hash_keep_mask(s1, m, 2 * h, p1, "cuda"), hdn / (1 - p1), torch.zeros(1, device="cuda"))
    hdn = hdn + (hdn.bfloat16().float() - hdn).detach()
    o = hdn @ w2.t() + b2
    if p2 > 0:
        o = torch.where(gemm.hash_keep_mask(s2, m, h, p2, "cuda"), o / (1 - p2), torch.zeros(1, device="cuda"))
    o = o + x2
    o.backward(dy.float())
    _close(y.detach(), o.detach(), torch.bfloat16)
    _close(x.grad, x2.grad, torch.bfloat16)
    for got, want in ((l1.weight.grad, w1.grad), (l2.weight.grad, w2.grad), (l1.bias.grad, b1.grad), (l2.bias.grad, b2.grad)):
        assert torch.allclose(got, want, atol=0.03 * float(want.abs().max()), rtol=5e-2)
    # the one-pass kernel by itself, and the epilogue's derivative against autograd of the exact GELU
    zz = (torch.randn(1001, 264, device="cuda") * 2).bfloat16()
    got = bnorm.gelu_dropout(zz, 1234, 0.3).float()
    want = torch.where(gemm.hash_keep_mask(1234, 1001, 264, 0.3, "cuda"), torch.nn.functional.gelu(zz.float()) / 0.7,
                       torch.zeros(1, device="cuda"))
    assert (got - want).abs().max() < 0.03 * max(1.0, float(want.abs().max()))
    a = torch.randn(777, 128, device="cuda").bfloat16()
    w = (torch.randn(256, 128, device="cuda") * 0.1).bfloat16()
    pre = (torch.randn(777, 256, device="cuda") * 1.5).bfloat16()
    got = gemm.gemm_tn(a, w, gelu_grad_of=pre).float()
    pf = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(pf).sum().backward()
    want = (a.float() @ w.float().t()) * pf.grad
    assert (got - want).abs().max() < 0.03 * max(1.0, float(want.abs().max()))
    gemm.check_status("cuda")


@pytest.mark.parametrize("act,residual,p1,p2,m", [("relu", True, 0.0, 0.0, 3000), ("gelu", True, 0.0, 0.0, 1111),
                                                  ("relu", False, 0.0, 0.0, 128 * 300 + 5), ("relu", True, 0.25, 0.1, 5000),
                                                  ("gelu", False, 0.3, 0.0, 257)])
def test_ffn_with_the_hidden_tile_on_chip_matches_reference(act, residual, p1, p2, m):
    """One-kernel feed-forward block (hidden tile in shared / tensor memory only) against a float32 restatement with the
    same hash dropout masks and the hidden tile rounded to bf16 as the kernel rounds it; ragged last tile, many tiles
    per CTA (both X buffers and all barrier phases in use), both activations, with and without the residual."""
    from budgetformer_b200.ops.ffn import ffn_onchip, onchip_supported
    torch.manual_seed(21)
    h = 128
    x = torch.randn(m, h, device="cuda").bfloat16()
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    assert onchip_supported(x, l1.weight, l2.weight)
    y = ffn_onchip(x, l1.weight, l1.bias, l2.weight, l2.bias, act=act, residual=residual, p1=p1, seed1=77, p2=p2, seed2=99)
    gemm.check_status("cuda")
    w1, w2 = l1.weight.detach().bfloat16().float(), l2.weight.detach().bfloat16().float()
    z = x.float() @ w1.t() + l1.bias.detach()
    hid = torch.relu(z) if act == "relu" else torch.nn.functional.gelu(z)
    if p1 > 0:
        hid = torch.where(gemm.hash_keep_mask(77, m, 2 * h, p1, "cuda"), hid / (1 - p1), torch.zeros(1, device="cuda"))
    hid = hid.bfloat16().float()
    o = hid @ w2.t() + l2.bias.detach()
    if p2 > 0:
        o = torch.where(gemm.hash_keep_mask(99, m, h, p2, "cuda"), o / (1 - p2), torch.zeros(1, device="cuda"))
    if residual:
        o = o + x.float()
    _close(y, o, torch.bfloat16)
    # the model-level entry takes this path for evaluation passes and agrees with the two-GEMM form it replaces
    from budgetformer_b200.ops import ffn as ffn_mod
    with torch.no_grad():
        a = ffn_mod.fused_ffn(x, l1.weight, l1.bias, l2.weight, l2.bias, act=act, residual=x if residual else None, training=False)
        old = ffn_mod.ONCHIP_FFN
        ffn_mod.ONCHIP_FFN = "0"
        try:
            b = ffn_mod.fused_ffn(x, l1.weight, l1.bias, l2.weight, l2.bias, act=act, residual=x if residual else None, training=False)
        finally:
            ffn_mod.ONCHIP_FFN = old
    assert (a.float() - b.float()).abs().max() < 0.06 * max(1.0, float(b.float().abs().max()))
    gemm.check_status("cuda")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("h", [64, 128])
@pytest.mark.parametrize("m", [1, 127, 128 * 3 + 33, 128 * 148 * 3 + 5])
def test_ffn_on_chip_widths_types_and_residuals(m, h, dtype):
    """Both widths and types, ReLU and GELU, each residual, with and without dropout and side outputs; fewer tiles than blocks, several a
    block, a ragged last one.  Hidden values against fp64 (one rounding to 8 or 11 bits, products added in fp32), the output against fp64
    products of the kernel's own hidden matrix."""
    from budgetformer_b200.ops.ffn import ffn_onchip, onchip_supported
    torch.manual_seed(m + h)
    f = 2 * h
    big = torch.randn(m, h + 8, device="cuda").to(dtype)
    x, other = big[:, :h], torch.randn(m, h, device="cuda").to(dtype)
    l1, l2 = torch.nn.Linear(h, f).cuda(), torch.nn.Linear(f, h).cuda()
    assert onchip_supported(x, l1.weight, l2.weight, other)
    w1, w2 = l1.weight.detach().to(dtype).double(), l2.weight.detach().to(dtype).double()
    b1, b2 = l1.bias.detach().double(), l2.bias.detach().double()
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    tiny = 0.0 if dtype == torch.bfloat16 else 2.0 ** -25
    near = lambda got, want, slack: ((got.double() - want).abs() <= half_ulp * (1 + 2.0 ** -7) * want.abs() + slack + tiny).all()
    zref = x.double() @ w1.t() + b1
    zslack = (x.double().abs() @ w1.abs().t() + 4) * h ** 0.5 * 2.0 ** -22 + 2.0 ** -20
    k1, k2 = gemm.hash_keep_mask(41, m, f, 0.25, "cuda"), gemm.hash_keep_mask(43, m, h, 0.125, "cuda")
    for act in ("relu", "gelu"):
        for p1, p2, res in ((0.0, 0.0, None), (0.25, 0.0, "x"), (0.25, 0.125, "other"), (0.0, 0.125, "other")):
            kw = dict(act=act, residual=res == "x", p1=p1, seed1=41, p2=p2, seed2=43, other=other if res == "other" else None)
            hid = torch.empty(m, f, device="cuda", dtype=dtype)
            side = dict(h_out=hid)
            if act == "gelu":
                side["z_out"] = torch.empty_like(hid)
            else:
                side["relu_bits_out"] = torch.empty(f // 16, m, device="cuda", dtype=torch.int16)
            y = ffn_onchip(x, l1.weight, l1.bias, l2.weight, l2.bias, **kw, **side)
            plain = ffn_onchip(x, l1.weight, l1.bias, l2.weight, l2.bias, **kw)
            gemm.check_status("cuda")
            if act == "gelu":
                assert near(side["z_out"], zref, zslack)
                want = torch.nn.functional.gelu(side["z_out"].double())
            else:
                want = zref.clamp(min=0)
            if p1 > 0:
                want = torch.where(k1, want / (1 - p1), 0.0)
            assert near(hid, want, 2 * zslack)
            if act == "relu":
                bits = torch.stack([(side["relu_bits_out"].int() >> i) & 1 for i in range(16)], 1).reshape(f, m).t().bool()
                sure = want.abs() > 4 * zslack
                assert torch.equal(bits & sure, (want > 0) & sure)
                assert torch.equal(y, plain)
            out = hid.double() @ w2.t() + b2
            if p2 > 0:
                out = torch.where(k2, out / (1 - p2), 0.0)
            if res is not None:
                out = out + (x if res == "x" else other).double()
            assert near(y, out, (hid.double().abs() @ w2.abs().t() + 8) * f ** 0.5 * 2.0 ** -22)
            _close(plain, out, dtype)


def test_ffn_on_chip_side_outputs_equal_the_two_gemm_form():
    """Training variant of the one-kernel block: the hidden matrix written from the on-chip operand and the ReLU bit mask
    equal what the first GEMM of the two-GEMM form writes (same masks, same rounding), over a ragged row count."""
    from budgetformer_b200.ops.ffn import ffn_onchip
    torch.manual_seed(8)
    m, h = 128 * 170 + 77, 128
    x = torch.randn(m, h, device="cuda").bfloat16()
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    w1, w2 = l1.weight.detach().bfloat16(), l2.weight.detach().bfloat16()
    bits_a = torch.zeros(2 * h // 16, m, dtype=torch.int16, device="cuda")
    h_a = gemm.gemm_tn(x, w1, l1.bias.detach(), "relu", dropout_p=0.2, dropout_seed=41, relu_bits_out=bits_a)
    y_a = gemm.gemm_tn(h_a, w2, l2.bias.detach(), None, dropout_p=0.1, dropout_seed=43, residual=x)
    h_b = torch.full((m, 2 * h), 9.0, device="cuda", dtype=torch.bfloat16)
    bits_b = torch.zeros_like(bits_a)
    y_b = ffn_onchip(x, l1.weight, l1.bias, l2.weight, l2.bias, act="relu", residual=True, p1=0.2, seed1=41, p2=0.1, seed2=43,
                     h_out=h_b, relu_bits_out=bits_b)
    gemm.check_status("cuda")
    assert (h_a.float() - h_b.float()).abs().max() < 2e-2 * max(1.0, float(h_a.float().abs().max()))
    mismatch = (bits_a != bits_b).float().mean()          # a sign can flip where a value rounds to or from zero
    assert float(mismatch) < 1e-3, float(mismatch)
    _close(y_b, y_a.float(), torch.bfloat16)


@pytest.mark.parametrize("act", ["relu", "gelu"])
@pytest.mark.parametrize("h", [64, 128])
def test_ffn_rows_that_overlap(h, act):
    """One row broadcast as the residual, and inputs and residuals whose rows overlap in memory, give what contiguous ones give, in
    evaluation and in training."""
    from budgetformer_b200.ops.ffn import fused_ffn
    torch.manual_seed(2)
    m = 200
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    flat = torch.randn(m * h, device="cuda").bfloat16()
    windows = flat.as_strided((m, h), (h // 2, 1))
    x = torch.randn(m, h, device="cuda").bfloat16()
    for inp, res in ((x, flat[:h].expand(m, h)), (x, windows), (windows, x), (windows, windows)):
        for grad in (False, True):
            with torch.set_grad_enabled(grad):
                got = fused_ffn(inp, l1.weight, l1.bias, l2.weight, l2.bias, act=act, residual=res)
                want = fused_ffn(inp.contiguous(), l1.weight, l1.bias, l2.weight, l2.bias, act=act, residual=res.contiguous())
            gemm.check_status("cuda")
            _close(got, want.float(), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gelu_carries_values_that_are_not_finite(dtype):
    """A NaN or an infinity in the bias reaches the activation as in PyTorch's GELU (NaN stays NaN, inf stays inf, -inf gives NaN), in the product's
    epilogue with and without its pre-activation and in the one-kernel block, and the block's output."""
    from budgetformer_b200.ops.ffn import ffn_onchip
    torch.manual_seed(3)
    m, h = 300, 64
    x = torch.randn(m, h, device="cuda").to(dtype)
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    with torch.no_grad():
        for col, bad in ((5, float("nan")), (70, float("inf")), (90, float("-inf")), (100, -1e4), (33, 1e4)):
            l1.bias[col] = bad
    b1, w1 = l1.bias.detach(), l1.weight.detach().to(dtype)
    want = torch.nn.functional.gelu(x.double() @ w1.double().t() + b1.double()).to(dtype)
    z, hid = (torch.empty(m, 2 * h, device="cuda", dtype=dtype) for _ in range(2))
    got = [gemm.gemm_tn(x, w1, b1, "gelu"), gemm.gemm_tn(x, w1, b1, "gelu", z_out=z)]
    y = ffn_onchip(x, l1.weight, l1.bias, l2.weight, l2.bias, act="gelu", residual=True, h_out=hid)
    plain = ffn_onchip(x, l1.weight, l1.bias, l2.weight, l2.bias, act="gelu", residual=True)
    assert z[:, 5].isnan().all() and z[:, 70].isinf().all()
    for t in got + [hid]:
        assert t[:, [5, 90]].isnan().all() and (t[:, 70] == float("inf")).all() and (t[:, 100] == 0).all()
        rest = [c for c in range(2 * h) if c not in (5, 70, 90)]
        # one rounding (8 or 11 bits) of a value within its fp32 sums, a second where the pre-activation is rounded first
        assert torch.allclose(t[:, rest].float(), want[:, rest].float(), rtol=2.0 ** -7, atol=2.0 ** -7)
    assert y.isnan().all() and plain.isnan().all()
    grad = gemm.gemm_tn(x, w1, gelu_grad_of=z)
    assert grad[:, 5].isnan().all()


@pytest.mark.parametrize("h,dtype,other", [(128, torch.bfloat16, True), (64, torch.bfloat16, True), (64, torch.bfloat16, False),
                                           (128, torch.float16, True), (64, torch.float16, False)])
def test_gelu_block_evaluates_what_it_trains(h, dtype, other):
    """Without gradients the block runs without side outputs; what it returns, with and without dropout, is what the training form
    returns, bit for bit: both take the activation of the rounded pre-activation."""
    from budgetformer_b200.ops.ffn import fused_ffn
    torch.manual_seed(h)
    x = torch.randn(1000, h, device="cuda").to(dtype)
    res = torch.randn(1000, h, device="cuda").to(dtype) if other else x
    l1, l2 = torch.nn.Linear(h, 2 * h).cuda(), torch.nn.Linear(2 * h, h).cuda()
    for p in (0.0, 0.25):
        got = []
        for grad in (True, False):
            torch.manual_seed(5)                              # the masks' seeds
            with torch.set_grad_enabled(grad):
                got.append(fused_ffn(x, l1.weight, l1.bias, l2.weight, l2.bias, act="gelu", residual=res, p1=p, p2=p))
        assert got[0].grad_fn is not None and got[1].grad_fn is None
        assert torch.equal(*got), p


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("h", [64, 128, 200, 512])
def test_layernorm_kernel(dtype, h):
    from budgetformer_b200.ops.norm import layer_norm
    torch.manual_seed(4)
    x = (torch.randn(3001, h, device="cuda") * 2 + 0.5).to(dtype).requires_grad_(True)
    ln = torch.nn.LayerNorm(h).cuda()
    with torch.no_grad():
        ln.weight.uniform_(0.5, 1.5)
        ln.bias.uniform_(-0.5, 0.5)
    y = layer_norm(x, ln.weight, ln.bias, ln.eps)
    dy = torch.randn_like(y)
    y.backward(dy)
    gw, gb = ln.weight.grad.clone(), ln.bias.grad.clone()
    ln.zero_grad()
    x2 = x.detach().float().requires_grad_(True)
    y2 = torch.nn.functional.layer_norm(x2, (h,), ln.weight, ln.bias, ln.eps)
    y2.backward(dy.float())
    tol = 3e-2 if dtype == torch.bfloat16 else 2e-4
    assert torch.allclose(y.float(), y2, atol=tol, rtol=tol)
    assert torch.allclose(x.grad.float(), x2.grad, atol=tol * max(1.0, float(x2.grad.abs().max())), rtol=tol)
    assert torch.allclose(gw, ln.weight.grad, atol=2e-2 * float(ln.weight.grad.abs().max()), rtol=2e-2)
    assert torch.allclose(gb, ln.bias.grad, atol=2e-2 * float(ln.bias.grad.abs().max()), rtol=2e-2)


def test_hash_dropout_matches_epilogue_mask():
    from budgetformer_b200.ops.norm import hash_dropout
    x = torch.ones(777, 96, device="cuda", dtype=torch.bfloat16)
    y = hash_dropout(x, 99, 0.3)
    keep = gemm.hash_keep_mask(99, 777, 96, 0.3, "cuda")
    assert torch.equal(y > 0, keep)
    assert abs(float(keep.float().mean()) - 0.7) < 0.02


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_column_sum_kernel(dtype):
    from budgetformer_b200.ops.norm import column_sum
    x = torch.randn(50001, 384, device="cuda").to(dtype)
    got = column_sum(x)
    want = x.double().sum(0)
    assert torch.allclose(got.double(), want, atol=0.2 if dtype == torch.bfloat16 else 2e-2, rtol=1e-3)
    view = x[:, 128:256]
    assert torch.allclose(column_sum(view).double(), view.double().sum(0), atol=0.2, rtol=1e-3)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("classes", [5, 40, 107])
def test_fused_nll_loss(dtype, classes):
    from budgetformer_b200.ops.loss import masked_nll
    torch.manual_seed(0)
    n = 5000
    logits = (torch.randn(n, classes, device="cuda") * 2).to(dtype).requires_grad_(True)
    y = torch.randint(0, classes, (n,), device="cuda")
    y[::7] = -1                                               # padded rows carry label -1 and are never selected
    idx = torch.nonzero(y >= 0).flatten()[::2].contiguous()
    loss = masked_nll(logits, y, idx)
    loss.backward()
    ref_in = logits.detach().float().requires_grad_(True)
    ref = torch.nn.functional.nll_loss(torch.log_softmax(ref_in[idx], 1), y[idx])
    ref.backward()
    # fp32: fast exp/log intrinsics and an atomic (order-dependent) sum over the rows
    assert abs(float(loss) - float(ref)) < (2e-2 if dtype == torch.bfloat16 else 1e-4)
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-5
    assert torch.allclose(logits.grad.float(), ref_in.grad, atol=tol * float(ref_in.grad.abs().max()) + 1e-9)


@pytest.mark.parametrize("n,n_dest,row0", [(384, 8, 0), (384, 4, 256), (384, 2, 0), (128, 8, 128), (128, 4, 0), (256, 8, 0)])
def test_gemm_routes_column_slices_to_destinations(n, n_dest, row0):
    """The fused all-to-all epilogue on one GPU: every destination is a local buffer here (peer pointers take the same
    path).  Slices of 48 / 96 / 16 / 32 columns use destination-wide staged panels, 192 the swizzled 64-column ones."""
    from budgetformer_b200.ops import _ext
    torch.manual_seed(1)
    m, k = 1000, 128
    cpd = n // n_dest
    x = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.1).bfloat16()
    bias = torch.randn(n, device="cuda")
    total_rows = row0 + m + 64
    outs = [torch.full((total_rows, cpd), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(n_dest)]
    _ext.load().gemm_tn(x, w, bias, 0, 0.0, 0, None, None, 1.0, False, [o.data_ptr() for o in outs], row0, cpd,
                        gemm.status_tensor("cuda"), None, None, 0)
    gemm.check_status("cuda")
    ref = x.float() @ w.float().t() + bias
    for d, o in enumerate(outs):
        got = o[row0:row0 + m].float()
        assert (got - ref[:, d * cpd:(d + 1) * cpd]).abs().max() < 0.06, d
        # rows outside this call's region stay untouched (the tail of the last row tile is clipped)
        assert bool((o[:row0] == 7.0).all()) and bool((o[row0 + m:] == 7.0).all()), d


def test_gemm_routes_slices_with_dropout_epilogue():
    """The d(context) push of the backward pass: no bias, the pre-projection dropout mask regenerated in the epilogue,
    16-column slices to 8 destinations (generic epilogue instance + destination-wide staged panels)."""
    from budgetformer_b200.ops import _ext
    torch.manual_seed(2)
    m, n, k, n_dest, p, seed = 777, 128, 128, 8, 0.25, 1234
    cpd = n // n_dest
    x = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.1).bfloat16()
    outs = [torch.zeros(m, cpd, device="cuda", dtype=torch.bfloat16) for _ in range(n_dest)]
    _ext.load().gemm_tn(x, w, None, 0, p, seed, None, None, 1.0, False, [o.data_ptr() for o in outs], 0, cpd,
                        gemm.status_tensor("cuda"), None, None, 0)
    gemm.check_status("cuda")
    keep = gemm.hash_keep_mask(seed, m, n, p, "cuda")
    ref = torch.where(keep, (x.float() @ w.float().t()) / (1 - p), torch.zeros(1, device="cuda"))
    got = torch.cat([o.float() for o in outs], 1)
    assert (got - ref).abs().max() < 0.06
    assert abs(float((got == 0).float().mean()) - p) < 0.03


def test_gemm_relu_bitmask_round_trip():
    """Forward epilogue writes one bit per element (result > 0 after ReLU and dropout); the backward epilogue masks with
    the bits: identical to masking with the stored activation."""
    torch.manual_seed(3)
    m, n, k = 1500, 256, 128
    x = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.1).bfloat16()
    bias = torch.randn(n, device="cuda") * 0.1
    bits = torch.zeros(n // 16, m, dtype=torch.int16, device="cuda")
    h = gemm.gemm_tn(x, w, bias, "relu", dropout_p=0.2, dropout_seed=99, relu_bits_out=bits)
    unpacked = ((bits.t().to(torch.int32).unsqueeze(-1) >> torch.arange(16, device="cuda")) & 1).reshape(m, n).bool()
    assert torch.equal(unpacked, h > 0)
    g = torch.randn(m, 128, device="cuda").bfloat16()
    w2 = (torch.randn(n, 128, device="cuda") * 0.1).bfloat16()
    a = gemm.gemm_tn(g, w2, relu_bits_in=bits, out_scale=1.25)
    b = gemm.gemm_tn(g, w2, relu_mask=h, out_scale=1.25)
    gemm.check_status("cuda")
    assert torch.equal(a, b)


@pytest.mark.parametrize("k", [72, 200, 272])
def test_gemm_ragged_k_panel_is_zero_filled(k):
    """K only has to keep rows 16-byte aligned: the last 64-element panel of both operands is zero-filled by TMA
    (the feature encoder runs with K = 272)."""
    torch.manual_seed(4)
    m, n = 1111, 128
    a = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn(n, k, device="cuda") / k ** 0.5).bfloat16()
    bias = torch.randn(n, device="cuda")
    out = gemm.gemm_tn(a, w, bias)
    gemm.check_status("cuda")
    _close(out, _ref(a, w, bias), torch.bfloat16)


@pytest.mark.parametrize("n_src,cps,n,row0,copy,extras", [
    (8, 16, 128, 0, True, True),        # context pull at 8 ranks, hidden 128: one K step per source
    (8, 48, 128, 512, True, False),     # dq|dk|dv pull at 8 ranks: three K steps per source, K = 384
    (4, 32, 128, 256, False, True),     # 4 ranks; no local copy (inference / recompute-free tiers)
    (2, 64, 128, 0, True, False),
    (2, 96, 64, 128, True, True),       # hidden 64 on 2 ranks: K = 192, a last stage of one panel
    (8, 32, 256, 1000, True, True),     # hidden 256 at 8 ranks: one 256-wide column chunk, so no tile is fetched twice
    (5, 16, 128, 64, True, False),      # K = 80: the last operand stage holds a single 16-column panel
])
def test_gemm_pulls_operand_column_slices_from_sources(n_src, cps, n, row0, copy, extras):
    """The fused heads->nodes all-to-all on one GPU: every source is a local buffer here (peer mappings take the same
    TMA path).  The gathered operand is checked through the product against an fp32 reference and, when a local copy is
    requested, bit for bit against the sources."""
    from budgetformer_b200.ops import _ext
    torch.manual_seed(11)
    m = 1000
    k = n_src * cps
    total_rows = row0 + m + 200                       # rows of other ranks follow this rank's block
    srcs = [torch.randn(total_rows, cps, device="cuda").bfloat16() for _ in range(n_src)]
    w = (torch.randn(n, k, device="cuda") / k ** 0.5).bfloat16()
    bias = torch.randn(n, device="cuda") if extras else None
    res = torch.randn(m, n, device="cuda").bfloat16() if extras else None
    out = torch.full((m, n), 3.0, device="cuda", dtype=torch.bfloat16)
    a_copy = torch.full((m, k), 5.0, device="cuda", dtype=torch.bfloat16) if copy else None
    _ext.load().gemm_tn_pull([s.data_ptr() for s in srcs], row0, cps, cps, m, w, a_copy, bias, 0.0, 0, res, 1.0, out,
                             gemm.status_tensor("cuda"))
    gemm.check_status("cuda")
    gathered = torch.cat([s[row0:row0 + m] for s in srcs], 1)
    ref = gathered.float() @ w.float().t()
    if extras:
        ref = ref + bias + res.float()
    assert (out.float() - ref).abs().max() < 0.06
    if copy:
        assert torch.equal(a_copy, gathered)


@pytest.mark.parametrize("m,n,k,bias", [
    (5000, 384, 128, True),      # packed q|k|v projection: three 128-feature tiles of dY
    (3333, 128, 128, True),      # output projection, ragged row count
    (4097, 256, 128, True),      # first FFN layer
    (2500, 128, 256, True),      # second FFN layer: two 128-feature chunks of X side by side, bias with the second
    (1111, 128, 272, True),      # feature encoder: three column chunks of X (128 + 128 + 16), bias rides with the last
    (777, 64, 128, True),        # readout: fewer than 128 features of dY (the tile's upper half is zero-filled)
    (50, 32, 64, True),          # fewer rows than one ring stage
    (200000, 128, 192, True),    # many row slices; chunks of 128 + 64 features
])
def test_weight_gradient_gemm_matches_fp32_reference(m, n, k, bias):
    """dW = dY^T X (+ column sums of dY) on the MN-major tcgen05 kernel against a float32 matmul of the same bf16
    operands.  fp32 accumulation in both: the difference is summation order."""
    torch.manual_seed(5)
    dy = torch.randn(m, n, device="cuda").bfloat16()
    x = torch.randn(m, k, device="cuda").bfloat16()
    dw, db = gemm.weight_grad(dy, x, bias)
    gemm.check_status("cuda")
    ref = dy.float().t() @ x.float()
    tol = 2e-3 * (m ** 0.5) + 1e-3
    assert dw.dtype == torch.float32 and dw.shape == (n, k)
    assert (dw - ref).abs().max() < tol, float((dw - ref).abs().max())
    if bias:
        assert (db - dy.float().sum(0)).abs().max() < tol
    else:
        assert db is None
    # bit-reproducible: slices are added in a fixed order
    dw2, _ = gemm.weight_grad(dy, x, bias)
    assert torch.equal(dw, dw2)


def test_weight_gradient_gemm_on_strided_views():
    """Operands that are column slices of wider matrices (row stride > width), as the packed q|k|v gradients are."""
    torch.manual_seed(6)
    m = 3000
    big = torch.randn(m, 512, device="cuda").bfloat16()
    dy, x = big[:, 128:256], big[:, 256:384]
    dw, db = gemm.weight_grad(dy, x, True)
    gemm.check_status("cuda")
    assert (dw - dy.float().t() @ x.float()).abs().max() < 0.2
    assert (db - dy.float().sum(0)).abs().max() < 0.2


@pytest.mark.parametrize("n_out,k", [(5, 128), (40, 128), (47, 256), (64, 128), (32, 64), (5, 32), (7, 16), (5, 8)])
def test_readout_linear_pads_narrow_outputs(n_out, k):
    """Output layers narrower than the kernels' 16-column granule run with zero rows appended to the weight: forward and
    all three gradients equal the float32 reference, down to 16 input features (one mostly zero-filled operand panel);
    inputs with fewer than 16 features fall back to the library."""
    torch.manual_seed(13)
    m = 2000
    x = torch.randn(m, k, device="cuda").bfloat16().requires_grad_(True)
    lin = torch.nn.Linear(k, n_out).cuda()
    y = gemm.readout_linear(x, lin.weight, lin.bias)
    assert y.shape == (m, n_out)
    dy = torch.randn(m, n_out, device="cuda").bfloat16()
    y.backward(dy)
    gemm.check_status("cuda")
    x2 = x.detach().float().requires_grad_(True)
    w2, b2 = lin.weight.detach().clone().requires_grad_(True), lin.bias.detach().clone().requires_grad_(True)
    ref = x2 @ w2.t() + b2
    ref.backward(dy.float())
    assert (y.float() - ref).abs().max() < 0.05
    assert (x.grad.float() - x2.grad).abs().max() < 0.05 * max(1.0, float(x2.grad.abs().max()))
    # the kernels leave fp32 gradients; the library fallback (k < 16) rounds them to bf16
    wtol = 2e-3 * m ** 0.5 + 1e-2 if k >= 16 else 2 ** -7 * float(w2.grad.abs().max())
    assert (lin.weight.grad - w2.grad).abs().max() < wtol
    assert (lin.bias.grad - b2.grad).abs().max() < (2e-3 * m ** 0.5 + 1e-2 if k >= 16 else 2 ** -7 * float(b2.grad.abs().max()) + 1e-2)
