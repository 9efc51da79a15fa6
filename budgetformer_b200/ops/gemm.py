"""Linear layers on the tcgen05 GEMMs (``csrc/gemm_tcgen05.cu``, ``csrc/gemm_dw_tcgen05.cu``).

``gemm_tn`` is the raw call ``C = A @ W.T`` with the fused epilogue; ``weight_grad`` is ``dW = dY^T X`` together
with the bias gradient (column sums of ``dY``) from one pass over the operands; ``fused_linear`` is the autograd
function used by the models on B200: forward, input gradient and weight gradient all run on the tcgen05 kernels.
Shapes the kernels do not cover (features not a multiple of 8 / 16, fp32 operands) fall back to PyTorch."""
from __future__ import annotations

import itertools
import threading
import weakref
from typing import Optional

import torch

from . import _ext

ACT = {None: 0, "none": 0, "relu": 1, "gelu": 2}
_STATUS = {}

# ---- operand copies of the weights ------------------------------------------------------------------------
# The kernels take weights in the activation dtype (and the input-gradient GEMM takes them transposed, the packed projection several
# in one).  Those copies only change when the weights do: they are kept per parameter and rebuilt when the parameter's version counter moves
# (in-place updates by PyTorch optimizers, ``load_state_dict``) or when an optimizer that writes the storage of its parameters directly
# announces a step (``ops.optim.FlatAdamW``: ``watch_weights``, ``weights_changed``).  A weight that belongs to no such optimizer may be
# written through ``.data`` by whatever runs beside one (a moving average of a model): any of their steps makes its copies stale.
#
# A copy is made on the stream that asks for it.  With it go the copies that the last announced step of the same optimizer made stale, if the
# step was announced on this stream, nothing wrote the weights after it, and no other stream has used the copies since they were last
# made: one launch (``csrc/param_kernels.cu``) in the place of one to three a copy.  A copy that another stream asks for waits there for its launch.
_WEIGHT_GEN = 0
_WEIGHT_COPIES = {}
_RECIPES = {}
_GROUPS = {}                                          # id of an optimizer's counter -> the recipes of its weights
_RECIPE_LOCK = threading.Lock()
_KIND = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


_OWNERS = {}                                          # id of a parameter -> (weak reference, counters of the optimizers that write it)
_STEPS = itertools.count(1)                           # never the same value twice, whichever optimizer it belongs to
_LAST_STEP = 0
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def watch_weights(params, counter: list) -> None:
    """``counter[0]`` changes whenever an optimizer writes ``params``, past their version counters maybe.  ``counter[1:]`` is filled in
    here: the stream of the last announced step, the device of the parameters, and their versions behind the step where it moves them."""
    for k in [k for k, (ref, _) in _OWNERS.items() if ref() is None]:
        del _OWNERS[k]
    counter[1:] = [None, None, None]
    for p in params:
        owner = _OWNERS.get(id(p))
        counters = owner[1] if owner is not None and owner[0]() is p else ()
        if all(c is not counter for c in counters):
            _OWNERS[id(p)] = (weakref.ref(p), counters + (counter,))
        if counter[2] is None and p.is_cuda:
            counter[2] = p.device.index


def watch_optimizer(optimizer) -> None:
    """``watch_weights`` for an optimizer of PyTorch, whose steps move the version counters: its steps announce themselves."""
    params = [p for g in optimizer.param_groups for p in g["params"]]
    counter = [0]
    watch_weights(params, counter)
    counter[3] = {}

    def announce(*_):
        weights_changed(counter, {id(p): p._version for p in params})

    optimizer.register_step_post_hook(announce)


def weights_changed(counter: Optional[list] = None, versions: Optional[dict] = None) -> None:
    """The weights watched with ``counter`` are written by what the current stream runs next, or have been by what it ran last where
    their ``versions`` are given; without a counter, any weight may have changed."""
    global _WEIGHT_GEN, _LAST_STEP
    if counter is not None:
        counter[0] = next(_STEPS)
        if versions is None:
            _LAST_STEP = counter[0]
        if len(counter) > 3 and counter[2] is not None:
            counter[1], counter[3] = _raw_stream(counter[2]), versions
    else:
        _WEIGHT_GEN += 1


def _counters(t: torch.Tensor) -> tuple:
    owner = _OWNERS.get(id(t))
    return owner[1] if owner is not None and owner[0]() is t else ()


def _only_counter(t: torch.Tensor) -> Optional[list]:
    counters = _counters(t)
    return counters[0] if len(counters) == 1 else None


def _stamp(srcs):
    out = [_WEIGHT_GEN]
    for t in srcs:
        owner = _OWNERS.get(id(t))                    # once a lookup of a copy: _counters without the calls
        if owner is None or owner[0]() is not t:
            steps = _LAST_STEP
        else:
            counters = owner[1]
            steps = counters[0][0]
            if len(counters) > 1:
                steps = max(c[0] for c in counters)
            if counters[0][3] is not None and steps < _LAST_STEP:      # whose optimizer writes through the version counters
                steps = _LAST_STEP
        out += (t._version, t.data_ptr(), steps)
    return out


class _Recipe:
    """A matrix made of blocks of fp32 matrices: ``blocks`` holds (source, first row, rows, columns, offset, row pitch, transposed).
    ``made`` is the copy: (stamp, tensor, stream, event behind its launch, list of the other streams that have waited for it)."""

    __slots__ = ("srcs", "blocks", "out_spec", "made", "used", "device", "counter")

    def __init__(self, srcs, blocks, out_spec):
        self.srcs = tuple(weakref.ref(t) for t in srcs)
        self.blocks, self.out_spec = blocks, out_spec
        self.made, self.used, self.counter = None, True, None
        self.device = srcs[0].device

    @property
    def out(self):
        return None if self.made is None else self.made[1]

    def sources(self):
        ts = [r() for r in self.srcs]
        return None if any(t is None for t in ts) else ts

    def take(self, made) -> torch.Tensor:
        """``made`` for the current stream."""
        _, out, stream, event, others = made
        now = _raw_stream(self.device.index)
        # while a graph is recorded, what was made before lies behind the synchronisation that the recording began with
        if now != stream and now not in others and not torch.cuda.is_current_stream_capturing():
            here = torch.cuda.current_stream(self.device)
            here.wait_event(event)
            out.record_stream(here)
            others.append(now)
        self.used = True
        return out


def _by_the_step(old, new, srcs, counter) -> bool:
    """Of two stamps of ``srcs``: nothing wrote them after the last step announced with ``counter``."""
    versions = counter[3] or {}
    return old[0] == new[0] and old[2::3] == new[2::3] and all(
        v == was or v == versions.get(id(t)) for v, was, t in zip(new[1::3], old[1::3], srcs))


def _rebuild(key, wanted: _Recipe, srcs, stamp) -> torch.Tensor:
    """Make ``wanted`` anew, and with it what its optimizer's last step made stale on this stream."""
    with _RECIPE_LOCK:
        stream = _raw_stream(wanted.device.index)
        # recorded launches have not run: what they make belongs to the graph alone, and nobody else may find it
        recording = torch.cuda.is_current_stream_capturing()
        todo = [(wanted, srcs, stamp)]
        if not recording:
            counter = _only_counter(srcs[0])
            if counter is not wanted.counter:
                _leave_group(key, wanted)
                if counter is not None:
                    wanted.counter = counter
                    _GROUPS.setdefault(id(counter), {})[key] = wanted
            if counter is not None and wanted.made is not None and counter[1] == stream and counter[2] == wanted.device.index:
                group, dead = _GROUPS[id(counter)], []
                for k, r in group.items():
                    made = r.made
                    if r is wanted or not r.used or made is None or made[2] != stream or made[4] or r.device != wanted.device:
                        continue
                    ts = r.sources()
                    if ts is None:
                        dead.append((k, r))
                        continue
                    now = _stamp(ts)
                    if (made[0] != now and _by_the_step(made[0], now, ts, counter) and all(_only_counter(t) is counter for t in ts)
                            and _plain_sources(ts)):
                        todo.append((r, ts, now))
                for k, r in dead:
                    _leave_group(k, r)
                    _RECIPES.pop(k, None)
        at, flat, items, outs = {}, [], [], []
        for i, (r, ts, _) in enumerate(todo):
            for t in ts:
                if id(t) not in at:
                    at[id(t)] = len(flat)
                    flat.append(t.detach())
            for blk in r.blocks:
                items.extend((at[id(ts[blk[0]])], blk[1], blk[2], blk[3], i, blk[4], blk[5], blk[6]))
            outs.extend(r.out_spec)
        made = _ext.load().weight_copies(flat, items, outs)
        _ext.count_launches((len(items) // 8 + 63) // 64)
        if recording:
            return made[0]
        event = torch.cuda.Event()
        event.record(torch.cuda.current_stream(wanted.device))
        for (r, _, now), out in zip(todo, made):
            r.made, r.used = (now, out, stream, event, []), r is wanted
        return made[0]


def _leave_group(key, r: _Recipe) -> None:
    if r.counter is not None:
        group = _GROUPS.get(id(r.counter), {})
        group.pop(key, None)
        if not group:
            _GROUPS.pop(id(r.counter), None)
        r.counter = None


def _plain_sources(srcs) -> bool:
    """fp32, contiguous and plain: what the copy kernel reads."""
    return all(t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() and t.numel() > 0 and t.device == srcs[0].device
               and not torch._C._functorch.is_functorch_wrapped_tensor(t) for t in srcs)


def recipe_copy(key, srcs, blocks, out_spec) -> torch.Tensor:
    """The matrix that ``blocks`` (a function that lists them) put together, kept under ``key`` until one of ``srcs`` changes."""
    r = _RECIPES.get(key)
    if r is None or any(ref() is not t for ref, t in zip(r.srcs, srcs)) or r.device != srcs[0].device:
        old, r = r, _Recipe(srcs, blocks(), out_spec)
        with _RECIPE_LOCK:
            if old is not None:
                _leave_group(key, old)
            _RECIPES[key] = r
            if len(_RECIPES) > 4096:                   # parameters of discarded models: drop what is dead
                for k, v in [(k, v) for k, v in _RECIPES.items() if v.sources() is None]:
                    _leave_group(k, _RECIPES.pop(k))
    stamp, made = _stamp(srcs), r.made
    if made is None or made[0] != stamp:
        return _rebuild(key, r, srcs, stamp)
    return r.take(made)


def operand_copy(weight: torch.Tensor, dtype, transpose: bool = False, index: Optional[torch.Tensor] = None,
                 tag: str = "") -> torch.Tensor:
    """``weight[index].to(dtype)`` (``.t()`` when ``transpose``), contiguous, cached until the weight changes."""
    key = (id(weight), dtype, bool(transpose), tag)
    stamp = _stamp((weight,))
    if index is None:
        r = _RECIPES.get(key)
        made = r.made if r is not None else None
        if made is not None and made[0] == stamp and r.srcs[0]() is weight:
            return r.take(made)                        # a forward pass asks this a dozen times: before any other look at the tensor
        # a tensor that is no parameter (a padded weight, made in every call) comes once: nothing to make beside it
        if isinstance(weight, torch.nn.Parameter) and weight.dim() == 2 and weight.is_leaf and dtype in _KIND and _plain_sources((weight,)):
            n, k = weight.shape
            return recipe_copy(key, (weight,), lambda: ((0, 0, n, k, 0, n if transpose else k, int(transpose)),),
                               (_KIND[dtype], k, n) if transpose else (_KIND[dtype], n, k))
    hit = _WEIGHT_COPIES.get(key)
    if hit is not None and hit[0] == stamp and hit[2]() is weight:
        return hit[1]
    w = weight.detach()
    if index is not None:
        w = w[index]
    w = w.to(dtype)
    w = w.t().contiguous() if transpose else w.contiguous()
    if weight.is_cuda and torch.cuda.is_current_stream_capturing():
        return w                                       # not computed yet
    _WEIGHT_COPIES[key] = (stamp, w, weakref.ref(weight))
    if len(_WEIGHT_COPIES) > 4096:                     # parameters of discarded models: drop what is dead
        for k in [k for k, v in _WEIGHT_COPIES.items() if v[2]() is None]:
            del _WEIGHT_COPIES[k]
    return w


def status_tensor(device) -> torch.Tensor:
    """Per-device int32[4] written by kernels whose bounded waits expired (0 = healthy)."""
    key = torch.device(device).index or 0
    t = _STATUS.get(key)
    if t is None:
        t = torch.zeros(4, dtype=torch.int32, device=device)
        _STATUS[key] = t
    return t


def check_status(device) -> None:
    """Host read of the status word; raises if any kernel gave up waiting."""
    t = _STATUS.get(torch.device(device).index or 0)
    if t is not None:
        code = int(t[0].item())
        if code != 0:
            t.zero_()
            raise RuntimeError(f"a device-side bounded wait expired (status {code}); results of that launch are invalid")


def supported(m: int, n: int, k: int, dtype) -> bool:
    return dtype in (torch.bfloat16, torch.float16) and m > 0 and k % 8 == 0 and k >= 16 and n % 16 == 0 and n >= 16


def gemm_tn(a: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, act: Optional[str] = None,
            dropout_p: float = 0.0, dropout_seed: int = 0, residual: Optional[torch.Tensor] = None,
            relu_mask: Optional[torch.Tensor] = None, out_scale: float = 1.0, out: Optional[torch.Tensor] = None,
            out_dtype: Optional[torch.dtype] = None, relu_bits_out: Optional[torch.Tensor] = None,
            relu_bits_in: Optional[torch.Tensor] = None, gelu_grad_of: Optional[torch.Tensor] = None,
            z_out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``act(dropout(a @ w.T * out_scale + bias)) [masked] + residual`` in one kernel.  ``relu_bits_out`` (int16
    ``[N / 16, M]``) receives one bit per element (result > 0); ``relu_bits_in`` zeroes the result where its bit is clear;
    ``gelu_grad_of`` (``[M, N]`` pre-activations) multiplies the result by ``gelu'(z)`` after the dropout mask - the
    hidden gradient of a GELU feed-forward block straight out of the GEMM; ``z_out`` (``[M, N]``, with ``act="gelu"`` and a bias) receives the
    pre-activation in its dtype, and the activation is taken of those rounded values."""
    if gelu_grad_of is not None:
        assert relu_mask is None, "one mask operand per call"
        relu_mask = gelu_grad_of
    ext = _ext.load()
    m, n = a.size(0), w.size(0)
    fp32_out = (out_dtype or (out.dtype if out is not None else a.dtype)) == torch.float32
    if out is None:
        out = torch.empty((m, n), dtype=torch.float32 if fp32_out else a.dtype, device=a.device)
    if m == 0:
        return out
    if bias is not None:
        bias = bias.float().contiguous()
        if bias.data_ptr() % 16:                      # the epilogue reads the bias with 16-byte loads
            bias = bias.clone()
    ext.gemm_tn(a, w, bias, ACT[act], float(dropout_p), int(dropout_seed),
                residual, relu_mask, float(out_scale), bool(fp32_out), [out.data_ptr()], 0, out.stride(0),
                status_tensor(a.device), relu_bits_out, relu_bits_in, 1 if gelu_grad_of is not None else 0, z_out)
    _ext.count_launches(1)
    return out


def weight_grad(dy: torch.Tensor, x: torch.Tensor, want_bias: bool = False):
    """``(dy.T @ x, dy.sum(0) or None)`` in fp32.  One tcgen05 kernel reads both operands once (MN-major tiles straight
    from the row-major matrices) and leaves per-row-slice partial tiles that a second kernel adds in a fixed order; the
    bias gradient is one more accumulator column of the same kernel.  Falls back to PyTorch for shapes outside the
    kernel's reach (features not a multiple of 8, operands that are not 16-bit)."""
    ext = _ext.load()
    m, n, k = dy.size(0), dy.size(1), x.size(1)
    ok = (dy.is_cuda and dy.dtype in (torch.bfloat16, torch.float16) and x.dtype == dy.dtype and m > 0
          and dy.stride(1) == 1 and x.stride(1) == 1 and (dy.stride(0) * 2) % 16 == 0 and (x.stride(0) * 2) % 16 == 0
          and dy.data_ptr() % 16 == 0 and x.data_ptr() % 16 == 0 and ext.gemm_dw_supported(m, n, k, False))
    if not ok:
        dw = torch.matmul(dy.t(), x).float()
        return dw, (dy.float().sum(0) if want_bias else None)
    fused_bias = bool(want_bias and ext.gemm_dw_supported(m, n, k, True))
    out = ext.gemm_dw(dy, x, fused_bias, status_tensor(dy.device))
    _ext.count_launches(3 if fused_bias else 2)
    db = out[1] if fused_bias else None
    if want_bias and db is None:
        from .norm import column_sum
        db = column_sum(dy)
    return out[0], db


def hash_keep_mask(seed: int, rows: int, cols: int, p: float, device) -> torch.Tensor:
    """The epilogue's dropout keep mask, restated in PyTorch (tests and the fallback path)."""
    r = torch.arange(rows, device=device, dtype=torch.int64)[:, None]
    c = torch.arange(cols, device=device, dtype=torch.int64)[None, :]
    x = (r * 0x9E3779B1 + c * 0x85EBCA77 + (int(seed) & 0xFFFFFFFF)) & 0xFFFFFFFF
    x = ((x ^ (x >> 16)) * 0x7FEB352D) & 0xFFFFFFFF
    x = ((x ^ (x >> 15)) * 0x846CA68B) & 0xFFFFFFFF
    x = x ^ (x >> 16)
    return x >= int(p * 4294967296.0)


class _FusedLinear(torch.autograd.Function):
    """y = residual + dropout(x W^T + b): one GEMM forward; input-gradient GEMM + weight-gradient GEMM backward."""

    @staticmethod
    def forward(ctx, x, weight, bias, residual, dropout_p, dropout_seed):
        w16 = operand_copy(weight, x.dtype)
        y = gemm_tn(x, w16, bias, None, dropout_p=dropout_p, dropout_seed=dropout_seed, residual=residual)
        ctx.cfg = (residual is not None, float(dropout_p), int(dropout_seed), weight.dtype, bias is not None)
        ctx.weight = weight
        ctx.save_for_backward(x)
        return y

    @staticmethod
    def backward(ctx, dy):
        from .norm import hash_dropout
        (x,) = ctx.saved_tensors
        has_res, p, seed, wdtype, has_bias = ctx.cfg
        dy = dy.contiguous()
        g = hash_dropout(dy, seed, p) if p > 0 else dy
        # dx = g @ W, expressed as g @ (W^T)^T; skipped for leaf inputs such as the feature matrix
        dx = None
        if ctx.needs_input_grad[0]:
            if supported(g.size(0), x.size(1), g.size(1), g.dtype):
                dx = gemm_tn(g, operand_copy(ctx.weight, x.dtype, transpose=True))
            else:                                      # fewer than 16 outputs (never through readout_linear, which pads)
                dx = torch.matmul(g, operand_copy(ctx.weight, x.dtype))
        dw, db = weight_grad(g, x, has_bias)
        return dx, dw.to(wdtype), (db.to(wdtype) if has_bias else None), (dy if has_res else None), None, None


def fused_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
                 residual: Optional[torch.Tensor] = None, dropout_p: float = 0.0, dropout_seed: int = 0) -> torch.Tensor:
    """2-D ``x``: ``residual + dropout(x @ weight.T + bias)``.  tcgen05 kernel when shape/dtype allow, else PyTorch."""
    if x.is_cuda and supported(x.size(0), weight.size(0), x.size(1), x.dtype) and x.stride(1) == 1 \
            and (x.stride(0) * 2) % 16 == 0 and x.data_ptr() % 16 == 0:
        return _FusedLinear.apply(x, weight, bias, residual, dropout_p, dropout_seed)
    y = torch.nn.functional.linear(x, weight.to(x.dtype), None if bias is None else bias.to(x.dtype))
    if dropout_p > 0:
        keep = hash_keep_mask(dropout_seed, y.size(0), y.size(1), dropout_p, y.device)
        y = torch.where(keep, y / (1.0 - dropout_p), torch.zeros_like(y))
    return y if residual is None else y + residual


def readout_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x @ weight.T + bias`` for the small output layers (h -> classes).  The tcgen05 kernels want the output width
    to be a multiple of 16: a narrower layer is run with zero rows appended to the weight (and zeros to the bias) and
    the extra columns are cut off again, so its forward, input gradient and weight gradient stay off the library GEMM
    (the kernels reduce over as few as 16 features: a narrower operand is one mostly zero-filled 64-wide panel).
    Inputs the kernels cannot take (fp32 activations, fewer than 16 input features) use ``torch.nn.functional.linear``."""
    n, k = weight.shape
    usable = (x.is_cuda and x.dim() == 2 and x.dtype in (torch.bfloat16, torch.float16) and k >= 16 and k % 8 == 0
              and x.stride(1) == 1 and (x.stride(0) * 2) % 16 == 0 and x.data_ptr() % 16 == 0)
    if not usable:
        return torch.nn.functional.linear(x, weight.to(x.dtype), None if bias is None else bias.to(x.dtype))
    pad = (-n) % 16
    if pad == 0:
        return fused_linear(x, weight, bias)
    w = torch.cat([weight, weight.new_zeros(pad, k)], 0)
    b = None if bias is None else torch.cat([bias, bias.new_zeros(pad)], 0)
    return fused_linear(x, w, b)[:, :n]


def plain_eager() -> bool:
    """False under tracing, compilation, ``torch.func`` transforms and forward-mode AD, which need PyTorch's own operators."""
    return not (torch.jit.is_tracing() or torch.compiler.is_compiling() or torch._C._are_functorch_transforms_active()
                or torch.autograd.forward_ad._current_level >= 0)


def plain_gradient(dy: torch.Tensor) -> bool:
    """False for the gradients of ``is_grads_batched`` (which set no transform that ``plain_eager`` could see), of transforms and
    of subclasses: a kernel would take their storage for the matrix they stand for."""
    return (type(dy) is torch.Tensor and not torch._C._functorch.is_legacy_batchedtensor(dy)
            and not torch._C._functorch.is_functorch_wrapped_tensor(dy) and plain_eager())


def _unit_columns(t: torch.Tensor) -> torch.Tensor:
    """``t`` with neighbouring columns next to each other.  One column has no neighbour: its stride is arbitrary (a transposed
    row), and ``contiguous()`` would leave it as it is."""
    return t if t.stride(1) == 1 or t.size(1) == 1 else t.contiguous()


class _LinearF32(torch.autograd.Function):
    """``torch.nn.functional.linear`` on fp32 with weight and bias gradient from ``csrc/linear_f32.cu``."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        ctx.save_for_backward(x, weight)
        ctx.has_bias = bias is not None
        return torch.nn.functional.linear(x, weight, bias)

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        n, k = weight.shape
        need_x, need_w, need_b = ctx.needs_input_grad
        dx = torch.matmul(dy, weight) if need_x else None
        dw = db = None
        if need_w or need_b:
            g, a = dy.reshape(-1, n), x.reshape(-1, k)
            if torch.is_grad_enabled() or not plain_gradient(dy):      # a second derivative, or many at once: PyTorch's operators
                return dx, g.t() @ a, g.sum(0) if ctx.has_bias else None
            flat = _ext.load().f32_weight_grad(_unit_columns(g), _unit_columns(a), ctx.has_bias)
            _ext.count_launches(2)
            dw, db = flat[:n * k].view(n, k), flat[n * k:] if ctx.has_bias else None
        return dx, dw, db


# Rows from which the gradient kernel is used; below, launches are all there is and both sides take two.
LINEAR_F32_MIN_ROWS = 128


def f32_gradient_pays(rows: int, n: int, k: int) -> bool:
    """Whether ``csrc/linear_f32.cu`` is the faster way to weight and bias gradient.  It adds 64 x 64 tiles with plain multiply-adds and
    splits the rows; the library splits its rows too little for few tiles, and has the better tile for many.  us, this kernel
    against the library's GEMM and column sum (outputs x features, rows):

    * up to 8 tiles: 64 x 64 13 / 28 at 128, 23 / 137 at 40 k, 63 / 307 at 200 k; 128 x 256 43 / 111 at 16 k, 525 / 677 at 262 k; 64 x 500
      394 / 503 at 200 k.  Widths that are no multiple of 4 take 4-byte copies: 64 x 269 647 / 710 at 262 k, 128 x 269 (10 tiles) 330 / 357
      at 66 k, 1279 / 828 at 262 k
    * 9 to 16 tiles: 192 x 192 839 / 1079 at 262 k; 256 x 256 17 / 32 at 1 k, 103 / 129 at 16 k, 372 / 376 at 66 k, 1448 / 926 at 262 k; 64 x 1000
      36 / 56 at 4 k, 103 / 100 at 16 k
    * up to 32 tiles: 64 x 1433 25 / 32 at 1 k, 58 / 58 at 4 k, 198 / 151 at 16 k; 320 x 320 157 / 189 at 16 k, 582 / 492 at 66 k; 512 x 256 56 / 68
      at 4 k, 188 / 159 at 16 k
    * more: 512 x 512 38 / 33 at 1 k, 864 / 510 at 40 k; 1024 x 1024 100 / 57 at 1 k
    * one output or feature (the library has a matrix-vector product): 1 x 64 13 / 19 at 4 k, 34 / 26 at 66 k; 1 x 256 21 / 18 at 8 k
    """
    if min(n, k) < 2:
        return rows <= 4096
    tiles = -(-n // 64) * -(-k // 64)
    return rows <= (1 << 40 if tiles <= 8 else 65536 if tiles <= 12 else 12288 if tiles <= 16 else 4096 if tiles <= 32 else 0)


def linear_f32(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``torch.nn.functional.linear``; on fp32 CUDA tensors outside autocast, where the kernel is the faster way
    (``f32_gradient_pays``), the weight and bias gradients come from this package's kernel.  Whoever lets fp32 products run in TF32
    gets the library's."""
    if (x.is_cuda and x.dtype == weight.dtype == torch.float32 and (bias is None or bias.dtype == torch.float32)
            and type(x) is torch.Tensor and x.dim() >= 2 and weight.device == x.device
            and weight.numel() > 0 and x.numel() >= LINEAR_F32_MIN_ROWS * weight.size(1)
            and f32_gradient_pays(x.numel() // weight.size(1), weight.size(0), weight.size(1))
            and torch.backends.cuda.matmul.fp32_precision != "tf32" and torch.is_grad_enabled() and weight.requires_grad
            and not torch.is_autocast_enabled("cuda") and plain_eager()):
        return _LinearF32.apply(x, weight, bias)
    return torch.nn.functional.linear(x, weight, bias)
