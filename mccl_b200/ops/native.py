"""autograd Functions over the native kernels (CUDA tensors only)."""
from __future__ import annotations

import functools
import itertools
import threading
import weakref

import torch
import torch.nn.functional as F

from .. import _C


def _bf16_weight(weight: torch.Tensor) -> torch.Tensor:
    """bf16 copy of an fp32 parameter: the trainer keeps one up to date (`_bf16`), else cast now."""
    w16 = getattr(weight, "_bf16", None)
    if w16 is not None:
        return w16
    if weight.dtype == torch.bfloat16:
        return weight
    return _C.cast_bf16(weight.detach().contiguous())


def _sink(p: torch.Tensor):
    """fp32 buffer a trainer wants this parameter's gradient written into (or None)."""
    return getattr(p, "_grad_sink", None)


def _notify(p: torch.Tensor) -> None:
    """Tells the trainer that p's gradient is complete (it was written in place, so autograd's
    own accumulation hook will not fire).  Parameters whose gradient has further contributions
    from autograd (tied embeddings) are marked `_shared_grad` and notified by autograd instead."""
    if getattr(p, "_shared_grad", False):
        return
    cb = getattr(p, "_grad_ready", None)
    if cb is not None:
        cb()


# Weight-gradient GEMMs have no consumer until the gradient is reduced or applied, so a trainer can give them a
# stream of their own: they then run beside the input-gradient chain and fill the SMs its small kernels leave idle.
_wgrad = {"stream": None, "pending": False, "side_ctas": 0, "main_ctas": 0}
_SIDE_COLSUM = __import__("os").environ.get("MCCL_SIDE_COLSUM", "1") != "0"


def set_wgrad_stream(stream, main_ctas: int = 0, side_ctas: int = 0) -> None:
    """Side stream for weight-gradient GEMMs that write into a trainer's gradient buffer (None: current stream).
    main_ctas / side_ctas: CTA caps of the GEMMs on the caller's stream and on the side stream while it is set
    (0: no cap); with caps that add up to the SM count a GEMM of one stream never waits for CTAs of the other."""
    _wgrad["stream"] = stream
    _wgrad["pending"] = False
    _wgrad["main_ctas"], _wgrad["side_ctas"] = main_ctas, side_ctas


def join_wgrad(stream=None) -> None:
    """Makes ``stream`` (default: the current one) wait for the weight gradients queued on the side stream."""
    _deferred.flush_all()
    _products.flush_all()
    s = _wgrad["stream"]
    if s is not None and _wgrad["pending"]:
        (stream if stream is not None else torch.cuda.current_stream()).wait_stream(s)


def _wgrad_gemm(a_mat: torch.Tensor, b_mat: torch.Tensor, sink: torch.Tensor, alpha=None) -> None:
    """sink += alpha * a_mat^T . b_mat (both [tokens, features]; alpha: a device scalar) on the weight-gradient stream."""
    s = _wgrad["stream"]
    if s is None:
        _C.gemm_bf16(a_mat, b_mat, None, "none", True, sink, True, True, True, alpha=alpha)
        return
    s.wait_stream(torch.cuda.current_stream())
    if _wgrad["side_ctas"]:
        _C.set_gemm_cta_limit(_wgrad["side_ctas"])
    with torch.cuda.stream(s):
        _C.gemm_bf16(a_mat, b_mat, None, "none", True, sink, True, True, True, alpha=alpha)
    if _wgrad["side_ctas"]:
        _C.set_gemm_cta_limit(_wgrad["main_ctas"])
    for t in (a_mat, b_mat) if alpha is None else (a_mat, b_mat, alpha):
        t.record_stream(s)
    _wgrad["pending"] = True


def _norm_param_grads(dyc, x, weight, mean, rstd, layernorm, wsink, bsink) -> bool:
    """dw / db of a norm on the weight-gradient stream; False when there is none (the caller then computes them in line)."""
    s = _wgrad["stream"] if _SIDE_COLSUM else None
    if s is None:
        return False
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        _C.norm_bwd(dyc, x, weight, mean, rstd, layernorm, wsink, bsink, True, None, 2)
    for t in (dyc, x, mean, rstd):
        t.record_stream(s)
    _wgrad["pending"] = True
    return True


def _wgrad_colsum(src: torch.Tensor, sink: torch.Tensor) -> None:
    """sink += column sums of src (a bias gradient), on the weight-gradient stream."""
    s = _wgrad["stream"] if _SIDE_COLSUM else None
    if s is None:
        _C.colsum_bf16(src, sink, True)
        return
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        _C.colsum_bf16(src, sink, True)
    src.record_stream(s)
    _wgrad["pending"] = True


def _gemm_ok(m: int, n: int, k: int) -> bool:
    return k % 64 == 0 and n % 8 == 0 and m > 0


def _linear_grads(dz, x2, w16, weight, need_dx: bool, need_dw: bool):
    """Gradients of x2 [M, K] and of weight [N, K] (None where it goes into the weight's own buffer), from dz [M, N]."""
    N, K = w16.shape
    M = x2.shape[0]
    dx = dw = None
    if need_dx:
        if _gemm_ok(M, K, N):
            # dx[M,K] = dz[M,N] · W[N,K]: W is the B operand stored [contraction, K], read MN-major
            dx, _ = _C.gemm_bf16(dz, w16, None, "none", False, None, False, False, True)
        else:
            dx = dz @ w16
    if need_dw:
        sink = _sink(weight)
        if _gemm_ok(N, K, M) and N % 8 == 0:
            # dW[N,K] = dz^T · x: both operands stored [tokens, features], read MN-major
            if sink is not None and _wgrad["stream"] is None:
                _products.add(dz, x2, sink, weight)
            elif sink is not None:
                _wgrad_gemm(dz, x2, sink)
                _notify(weight)
            else:
                dw, _ = _C.gemm_bf16(dz, x2, None, "none", True, None, False, True, True)
        else:
            dw = (dz.t() @ x2).float()
    return dx, dw


class LinearFn(torch.autograd.Function):
    """y = act(x @ W^T + b); W [N, K] fp32 master, x [..., K] bf16."""

    @staticmethod
    def forward(ctx, x, weight, bias, act, residual=None):
        K, N = weight.shape[1], weight.shape[0]
        x2 = x.reshape(-1, K)
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        M = x2.shape[0]
        w16 = _bf16_weight(weight)
        ctx.act, ctx.has_bias, ctx.native = act, bias is not None, _gemm_ok(M, N, K)
        res2 = None
        if residual is not None:
            res2 = residual.reshape(-1, N)
            if not res2.is_contiguous():
                res2 = res2.contiguous()
        ctx.has_residual = residual is not None
        if ctx.native:
            y, z = _C.gemm_bf16(x2, w16, bias, act, False, None, False, False, False, res2)
        else:
            z = F.linear(x2, w16, None if bias is None else bias.to(x2.dtype))
            y = F.gelu(z) if act == "gelu" else z
            z = z if act == "gelu" else None
            if res2 is not None:
                y = y + res2
        ctx.save_for_backward(x2, w16, z if z is not None else x2.new_empty(0))
        ctx.weight, ctx.bias = weight, bias
        return y.view(*x.shape[:-1], N)

    @staticmethod
    def backward(ctx, dy):
        x2, w16, z = ctx.saved_tensors
        weight = ctx.weight
        N, K = w16.shape
        M = x2.shape[0]
        dy2 = dy.reshape(-1, N)
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dz = _C.gelu_bwd(dy2, z) if ctx.act == "gelu" else dy2
        db = None
        dx, dw = _linear_grads(dz, x2, w16, weight, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        if dx is not None:
            dx = dx.view(*dy.shape[:-1], K)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            bsink = _sink(ctx.bias)
            if N % 8 == 0:
                if bsink is not None:
                    _wgrad_colsum(dz, bsink)
                    _notify(ctx.bias)
                else:
                    db = _C.colsum_bf16(dz)
            else:
                db = dz.sum(0, dtype=torch.float32)
        dres = dy if ctx.has_residual else None
        return dx, dw, db, None, dres


class MlpGeluFn(torch.autograd.Function):
    """y = gelu(x @ W1^T + b1) @ W2^T + b2 (+ residual) as one autograd node, so that backward can fuse across
    the two layers: the first GEMM's epilogue saves gelu'(z) next to gelu(z) (they share the erf), and the
    input-gradient GEMM of the second layer multiplies by it in its epilogue and writes dz directly, so there is
    no separate GELU-backward pass over the [tokens, d_ff] tensor.  (Evaluating erf and exp in the backward
    epilogue instead was measured slower than the separate kernel: four epilogue warps per SM are too few for it.)"""

    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, residual=None):
        D, FF = w1.shape[1], w1.shape[0]
        x2 = x.reshape(-1, D)
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        w1_16, w2_16 = _bf16_weight(w1), _bf16_weight(w2)
        h, z = _C.gemm_bf16(x2, w1_16, b1, "gelu_d")   # z holds gelu'(pre-activation)
        res2 = None
        if residual is not None:
            res2 = residual.reshape(-1, w2.shape[0])
            if not res2.is_contiguous():
                res2 = res2.contiguous()
        y, _ = _C.gemm_bf16(h, w2_16, b2, "none", False, None, False, False, False, res2)
        ctx.save_for_backward(x2, w1_16, w2_16, z, h)
        ctx.params = (w1, b1, w2, b2)
        ctx.has_residual = residual is not None
        return y.view(*x.shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w1_16, w2_16, z, h = ctx.saved_tensors
        w1, b1, w2, b2 = ctx.params
        dy2 = dy.reshape(-1, w2_16.shape[0])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        # second layer: dz = (dy . W2) * gelu'(pre-activation) in one kernel; dW2 = dy^T . h; db2 = column sums of dy
        dz, _ = _C.gemm_bf16(dy2, w2_16, None, "none", False, None, False, False, True, None, z)
        # the input gradient first: every reader of this node's weights is queued before a parameter is reported
        # complete (a trainer may start that parameter's optimizer update on another stream as soon as it is)
        dx = None
        if ctx.needs_input_grad[0]:
            dx, _ = _C.gemm_bf16(dz, w1_16, None, "none", False, None, False, False, True)
            dx = dx.view(*dy.shape[:-1], w1_16.shape[1])
        grads = {}
        for name, (w, a_mat, b_mat) in (("w2", (w2, dy2, h)), ("w1", (w1, dz, x2))):
            sink = _sink(w)
            if sink is not None:
                _wgrad_gemm(a_mat, b_mat, sink)
                _notify(w)
                grads[name] = None
            else:
                grads[name], _ = _C.gemm_bf16(a_mat, b_mat, None, "none", True, None, False, True, True)
        for name, (b, src) in (("b2", (b2, dy2)), ("b1", (b1, dz))):
            if b is None:
                grads[name] = None
                continue
            bsink = _sink(b)
            if bsink is not None:
                _wgrad_colsum(src, bsink)
                _notify(b)
                grads[name] = None
            else:
                grads[name] = _C.colsum_bf16(src)
        return dx, grads["w1"], grads["b1"], grads["w2"], grads["b2"], (dy if ctx.has_residual else None)


class CausalAttentionFn(torch.autograd.Function):
    """Causal self-attention on the output of the fused QKV projection, viewed as [B, S, 3, H, 64]: one kernel
    forward, one backward, both on the tcgen05 tensor cores; the gradient comes back for the whole qkv tensor, so
    no slices, transposes or concatenations surround the kernels."""

    @staticmethod
    def forward(ctx, qkv, scale):
        q5 = qkv if qkv.is_contiguous() else qkv.contiguous()
        o, lse = _C.attn_fwd(q5, scale)
        ctx.save_for_backward(q5, o, lse)
        ctx.scale = scale
        return o

    @staticmethod
    def backward(ctx, d_o):
        q5, o, lse = ctx.saved_tensors
        d = d_o if d_o.is_contiguous() else d_o.contiguous()
        return _C.attn_bwd(q5, o, d, lse, ctx.scale), None


class DecoderLayerFn(torch.autograd.Function):
    """A whole pre-LayerNorm GELU decoder layer as one autograd node (csrc/bindings/bind_layers.cpp).  params: weight and bias
    of first norm, qkv, output projection, second norm, up and down projection."""

    MATRICES = (2, 4, 8, 10)

    @staticmethod
    def forward(ctx, x, heads, eps, *params):
        w = list(params)
        todo = []
        for i in DecoderLayerFn.MATRICES:
            w16 = getattr(w[i], "_bf16", None)   # a trainer keeps one up to date
            if w16 is None:
                todo.append(i)
            else:
                w[i] = w16
        if todo:
            for i, w16 in zip(todo, _C.cast_many([w[i] for i in todo])):
                w[i] = w16
        B, S = x.shape[0], x.shape[1]
        out, slab = _C.decoder_layer_fwd(x, w, B, S, heads, eps)
        ctx.save_for_backward(x, slab, *w)
        ctx.params, ctx.heads = params, heads
        return out

    @staticmethod
    def backward(ctx, dout):
        x, slab, *w = ctx.saved_tensors
        params = ctx.params
        sinks = [getattr(p, "_grad_sink", None) for p in params]
        direct = all(s is not None for s in sinks)
        dout = dout if dout.is_contiguous() else dout.contiguous()
        B, S = x.shape[0], x.shape[1]
        dx, grads, between = _C.decoder_layer_bwd(dout, x, slab, w, sinks if direct else [], B, S, ctx.heads, direct)
        if not direct:
            return (dx, None, None, *grads)
        _deferred.add((dout, slab, between, sinks), (B, S, ctx.heads), params, x.device)
        return (dx, None, None) + (None,) * len(params)


class _Entry:
    """Products of one backward pass that wait for others: like ones only, on one stream."""

    __slots__ = ("kind", "stream", "items", "params", "size", "__weakref__")

    def __init__(self, kind, stream):
        self.kind, self.stream = kind, stream
        self.items, self.params, self.size = [], [], 0.0


class _Shared:
    """Weight gradients that go straight into a trainer's buffers, kept back until several can share a launch.  Flushed at the end
    of backward at the latest (by an engine callback), and before anybody looks at the gradients of a bucket.  Where peers wait
    for them (`_grad_awaited`) none is kept back: a bucket's collective starts with its last gradient, and the gain was measured
    on one GPU only.

    The callback owns the entry and this table only knows it: the engine drops its callbacks when a pass fails, and what
    was kept back goes with them instead of joining the next pass's products."""

    def __init__(self):
        self._lock = threading.Lock()
        self._pending = weakref.WeakValueDictionary()   # (device, backward pass) -> _Entry

    def _enter(self, device, kind, item, params, size) -> _Entry:
        """Adds an item to the current pass's entry; one of another kind is flushed first."""
        key = (device, torch._C._current_graph_task_id())
        stream = torch.cuda.current_stream(device)
        entry = self._pending.get(key)
        if entry is not None and (entry.kind != kind or entry.stream != stream):
            self._flush(entry)
            entry = None
        if entry is None:
            entry = _Entry(kind, stream)
            torch.autograd.Variable._execution_engine.queue_callback(functools.partial(self._flush, entry))
            self._pending[key] = entry
        with self._lock:
            entry.items.append(item)
            entry.params.append(params)
            entry.size += size
        if any(getattr(p, "_grad_awaited", False) for p in params):
            self._flush(entry)
        return entry

    def _flush(self, entry) -> None:
        with self._lock:
            items, params = entry.items, entry.params
            entry.items, entry.params, entry.size = [], [], 0.0
        if not items:
            return
        with torch.cuda.stream(entry.stream):
            self._launch(entry.kind, items)
            for p in itertools.chain.from_iterable(params):
                _notify(p)

    def flush_all(self) -> None:
        for entry in list(self._pending.values()):
            self._flush(entry)


class _Deferred(_Shared):
    """Weight gradients of decoder layers: a layer's four products fill the SMs for 20 us and pay 8 us of set-up, first loads and
    last epilogue, so at 4096 tokens four layers together take 23 us each instead of 25, at 1600 tokens 12 instead of 18, and a
    small model's 2 instead of 6."""

    #: multiply-adds that keep the GPU busy for some 60 us: enough for the fixed part to be small
    ENOUGH = 5e10
    MOST = 4

    def add(self, item, sizes, params, device) -> None:
        work = sizes[0] * sizes[1] * float(sum(item[3][i].numel() for i in DecoderLayerFn.MATRICES))
        entry = self._enter(device, (sizes, item[3][8].shape), item, params[::-1], work)
        if len(entry.items) >= self.MOST or entry.size >= self.ENOUGH:
            self._flush(entry)

    def _launch(self, kind, items) -> None:
        _C.decoder_layer_wgrads(items, *kind[0])


_deferred = _Deferred()


class _Products(_Shared):
    """Weight gradients of single linear layers.  One whose tiles leave half the SMs idle waits for the next ones over the same
    tokens and shares a launch with them (1024 x 1024 and 3072 x 1024 over 4096 tokens: two launches of 28 and 33 us beside the
    optimizer, one of 35)."""

    @staticmethod
    def limits():
        """(tiles of 256 x 256 up to which a product waits: half of what the SMs that products may use work on at a time; tiles
        beyond which one joins none that waits: seven eighths, 64 on 148 SMs)."""
        sms, cap = _C.gemm_sm_count(), _C.gemm_cta_limit()
        pairs = (min(sms, cap) if cap > 0 else sms) // 2
        return pairs // 2, pairs * 7 // 8

    def add(self, dz, x2, sink, weight) -> None:
        device, tokens = dz.device, dz.shape[0]
        tiles = -(-dz.shape[1] // 256) * -(-x2.shape[1] // 256)
        small, most = self.limits()
        entry = self._pending.get((device, torch._C._current_graph_task_id()))
        waiting = entry is not None and entry.items and entry.kind == tokens and entry.stream == torch.cuda.current_stream(device)
        if tiles > (most if waiting else small) or (not waiting and not dz.is_contiguous()):
            if entry is not None:
                self._flush(entry)
            _wgrad_gemm(dz, x2, sink)
            _notify(weight)
            return
        entry = self._enter(device, tokens, (dz.contiguous(), x2, sink), (weight,), tiles)
        if entry.size > small or len(entry.items) >= 4:
            self._flush(entry)

    def _launch(self, kind, items) -> None:
        _C.gemm_group(items, True)


_products = _Products()


class RopeQkvFn(torch.autograd.Function):
    """Fused QKV projection output [B, S, 3, H, hd] -> rotated q, rotated k, v, each [B, H, S, hd] (views).  One kernel
    each way: the backward turns dq and dk back and gathers all three into the gradient of the whole projection."""

    @staticmethod
    def forward(ctx, qkv, cos, sin):
        q5 = qkv if qkv.is_contiguous() else qkv.contiguous()
        qk = _C.rope_qk_fwd(q5, cos, sin)
        ctx.tables = (cos, sin)
        return qk[:, :, 0].transpose(1, 2), qk[:, :, 1].transpose(1, 2), q5[:, :, 2].transpose(1, 2)

    @staticmethod
    def backward(ctx, dq, dk, dv):
        def usable(g):
            return g if g.stride(3) == 1 and all(s % 8 == 0 for s in g.stride()[:3]) and g.data_ptr() % 16 == 0 else g.contiguous()
        return _C.rope_qkv_bwd(usable(dq), usable(dk), usable(dv), *ctx.tables), None, None


class SwigluFn(torch.autograd.Function):
    """silu(gate) * up for [..., 2 F] = [gate | up], one kernel each way."""

    @staticmethod
    def forward(ctx, gu):
        g2 = gu if gu.is_contiguous() else gu.contiguous()
        ctx.save_for_backward(g2)
        return _C.swiglu_fwd(g2)

    @staticmethod
    def backward(ctx, dh):
        (gu,) = ctx.saved_tensors
        return _C.swiglu_bwd(dh if dh.is_contiguous() else dh.contiguous(), gu)


class MlpSwigluFn(torch.autograd.Function):
    """y = (silu(gate) * up) @ W2^T (+ residual), [gate | up] = x @ W1^T, as one autograd node: the activation is the first
    product's epilogue, its backward that of the second product's input gradient."""

    @staticmethod
    def forward(ctx, x, w1, w2, residual=None):
        x2 = x.reshape(-1, w1.shape[1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        w1_16, w2_16 = _bf16_weight(w1), _bf16_weight(w2)
        h, gu = _C.gate_up_swiglu(x2, w1_16)
        res2 = None
        if residual is not None:
            res2 = residual.reshape(-1, w2.shape[0])
            if not res2.is_contiguous():
                res2 = res2.contiguous()
        y, _ = _C.gemm_bf16(h, w2_16, None, "none", False, None, False, False, False, res2)
        ctx.save_for_backward(x2, w1_16, w2_16, gu, h)
        ctx.params = (w1, w2)
        ctx.has_residual = residual is not None
        return y.view(*x.shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w1_16, w2_16, gu, h = ctx.saved_tensors
        w1, w2 = ctx.params
        dy2 = dy.reshape(-1, w2_16.shape[0])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dgu = _C.down_swiglu_bwd(dy2, w2_16, gu)
        # each weight's gradient once nothing reads the weight any more (see MlpGeluFn)
        _, dw2 = _linear_grads(dy2, h, w2_16, w2, False, ctx.needs_input_grad[2])
        dx, dw1 = _linear_grads(dgu, x2, w1_16, w1, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        if dx is not None:
            dx = dx.view(*dy.shape[:-1], x2.shape[1])
        return dx, dw1, dw2, (dy if ctx.has_residual else None)


class NormFn(torch.autograd.Function):
    """LayerNorm (bias given) or RMSNorm (bias None) over the last dimension; fp32 weight / bias."""

    @staticmethod
    def forward(ctx, x, weight, bias, eps):
        xc = x if x.is_contiguous() else x.contiguous()
        y, mean, rstd = _C.norm_fwd(xc, weight, bias, eps)
        ctx.save_for_backward(xc, weight, mean, rstd)
        ctx.layernorm = bias is not None
        ctx.weight, ctx.bias = weight, bias
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, mean, rstd = ctx.saved_tensors
        dyc = dy if dy.is_contiguous() else dy.contiguous()
        wsink, bsink = _sink(ctx.weight), (_sink(ctx.bias) if ctx.bias is not None else None)
        if wsink is not None and (not ctx.layernorm or bsink is not None):
            # the sinks were zeroed at the start of the step; the kernel adds into them
            side = _norm_param_grads(dyc, x, weight, mean, rstd, ctx.layernorm, wsink, bsink)
            dx, _, _ = _C.norm_bwd(dyc, x, weight, mean, rstd, ctx.layernorm, wsink, bsink, True, None, 1 if side else 3)
            _notify(ctx.weight)
            if ctx.bias is not None:
                _notify(ctx.bias)
            return dx, None, None, None
        dx, dw, db = _C.norm_bwd(dyc, x, weight, mean, rstd, ctx.layernorm)
        return dx, dw, db, None


class NormResidualFn(torch.autograd.Function):
    """Norm of a tensor that also continues as a residual: returns ``(norm(x), x)``.  In backward the
    gradient that comes back along the residual is added inside the norm-backward kernel (before its
    single rounding to bf16) instead of by a separate add kernel."""

    @staticmethod
    def forward(ctx, x, weight, bias, eps):
        xc = x if x.is_contiguous() else x.contiguous()
        y, mean, rstd = _C.norm_fwd(xc, weight, bias, eps)
        ctx.save_for_backward(xc, weight, mean, rstd)
        ctx.layernorm = bias is not None
        ctx.weight, ctx.bias = weight, bias
        return y, xc.view_as(xc)

    @staticmethod
    def backward(ctx, dy, dres):
        x, weight, mean, rstd = ctx.saved_tensors
        if dy is None:
            return dres, None, None, None
        dyc = dy if dy.is_contiguous() else dy.contiguous()
        add = None if dres is None else (dres if dres.is_contiguous() else dres.contiguous())
        wsink, bsink = _sink(ctx.weight), (_sink(ctx.bias) if ctx.bias is not None else None)
        if wsink is not None and (not ctx.layernorm or bsink is not None):
            side = _norm_param_grads(dyc, x, weight, mean, rstd, ctx.layernorm, wsink, bsink)
            dx, _, _ = _C.norm_bwd(dyc, x, weight, mean, rstd, ctx.layernorm, wsink, bsink, True, add, 1 if side else 3)
            _notify(ctx.weight)
            if ctx.bias is not None:
                _notify(ctx.bias)
            return dx, None, None, None
        dx, dw, db = _C.norm_bwd(dyc, x, weight, mean, rstd, ctx.layernorm, None, None, False, add)
        return dx, dw, db, None


class LinearCrossEntropyFn(torch.autograd.Function):
    """mean CE(h @ W^T, targets).  The backward of the loss with respect to the logits is
    produced in the same pass that computes the loss, in place of the logits, for an upstream
    gradient of one; the products of backward multiply by the one that comes."""

    @staticmethod
    def forward(ctx, h, weight, targets):
        T, D = h.shape
        V = weight.shape[0]
        hc = h if h.is_contiguous() else h.contiguous()
        w16 = _bf16_weight(weight)
        if _gemm_ok(T, V, D):
            logits, _ = _C.gemm_bf16(hc, w16)
        else:
            logits = F.linear(hc, w16)
        loss_rows = _C.ce_fwd_bwd(logits, targets.contiguous(), 1.0 / T)
        ctx.save_for_backward(hc, w16, logits)   # logits now hold d(loss)/d(logits)
        ctx.weight = weight
        return _C.mean_f32(loss_rows)

    @staticmethod
    def backward(ctx, gout):
        h, w16, dlogits = ctx.saved_tensors
        weight = ctx.weight
        T, D = h.shape
        V = w16.shape[0]
        up = gout.float().contiguous()
        dh = dw = None
        if ctx.needs_input_grad[0]:
            if _gemm_ok(T, D, V):
                dh, _ = _C.gemm_bf16(dlogits, w16, None, "none", False, None, False, False, True, alpha=up)
            else:
                dh = ((dlogits @ w16).float() * up).to(h.dtype)
        if ctx.needs_input_grad[1]:
            sink = _sink(weight)
            if _gemm_ok(V, D, T) and V % 8 == 0:
                if sink is not None:
                    _wgrad_gemm(dlogits, h, sink, up)
                    _notify(weight)
                else:
                    dw, _ = _C.gemm_bf16(dlogits, h, None, "none", True, None, False, True, True, alpha=up)
            else:
                dw = (dlogits.t() @ h).float() * up
        return dh, dw, None


class EmbeddingFn(torch.autograd.Function):
    """bf16(tok[ids] + pos[position]) in one kernel; the backward adds the output gradient into the
    fp32 gradient buffers of both tables (the trainer's sinks when there are any) with vector atomics,
    so no sort, no dense zero-filled intermediate and no autograd accumulation step is needed."""

    @staticmethod
    def forward(ctx, ids, tok, pos, seq):
        flat = ids.reshape(-1).contiguous()
        y = _C.embed_fwd(flat, tok.detach(), None if pos is None else pos.detach(), seq)
        ctx.save_for_backward(flat)
        ctx.tok, ctx.pos, ctx.seq = tok, pos, seq
        return y.view(*ids.shape, tok.shape[1])

    @staticmethod
    def backward(ctx, dy):
        (flat,) = ctx.saved_tensors
        tok, pos, seq = ctx.tok, ctx.pos, ctx.seq
        dyc = dy.reshape(-1, tok.shape[1])
        if not dyc.is_contiguous():
            dyc = dyc.contiguous()
        tsink = _sink(tok)
        psink = _sink(pos) if pos is not None else None
        dtok = tsink if tsink is not None else torch.zeros_like(tok, dtype=torch.float32)
        dpos = None
        if pos is not None:
            dpos = psink if psink is not None else torch.zeros_like(pos, dtype=torch.float32)
        _C.embed_bwd(flat, dyc, dtok, dpos, seq)
        # this is the last contribution to a tied table's gradient, so it is the one that reports it
        for p, sink in ((tok, tsink), (pos, psink)):
            if p is not None and sink is not None:
                cb = getattr(p, "_grad_ready", None)
                if cb is not None:
                    cb()
        return None, (None if tsink is not None else dtok), (None if pos is None or psink is not None else dpos), None

