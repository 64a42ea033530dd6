"""Decoder-only transformer family.

The reference's headline numbers are DDP samples/s on a 70M and a 110M decoder
(README.md:44-54; the training script itself is not in its tree, only a toy
model: examples/ddp_utils.py:41-147).  The architectures here are the ones the
baseline configurations spell out:

  70m   d_model 512,  16 layers,  8 heads, FFN 2048 GELU,   pre-LayerNorm, learned positions, vocab 32000, tied
  110m  d_model 768,  12 layers, 12 heads, FFN 3072 GELU,   pre-LayerNorm, learned positions, vocab 32000, tied
  1.3b  d_model 2048, 24 layers, 16 heads, FFN 8192 SwiGLU, RMSNorm, RoPE, vocab 32000

`Decoder` is a plain ``nn.Module`` (fp32 master parameters) whose forward runs
in bf16.  On a CUDA device its matmuls, normalisations, activation and loss go
through this package's sm_100a operators (``mccl_b200.ops``); with
``native=False`` or on CPU the same math runs on stock PyTorch operators, which
is also the numerics reference in the tests.
"""
from __future__ import annotations

import dataclasses
import itertools
import math
import operator
import os
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F


@dataclasses.dataclass
class DecoderConfig:
    vocab: int = 32000
    d_model: int = 512
    n_layers: int = 16
    n_heads: int = 8
    d_ff: int = 2048
    max_seq: int = 256
    act: str = "gelu"          # "gelu" | "swiglu"
    norm: str = "layernorm"    # "layernorm" | "rmsnorm"
    pos: str = "learned"       # "learned" | "rope"
    tied: bool = True
    eps: float = 1e-5

    @property
    def head_dim(self) -> int:
        return self.d_model // self.n_heads

    def param_count(self) -> int:
        ff = (3 if self.act == "swiglu" else 2) * self.d_model * self.d_ff
        attn = 4 * self.d_model * self.d_model
        per_layer = ff + attn
        emb = self.vocab * self.d_model * (1 if self.tied else 2)
        pos = self.max_seq * self.d_model if self.pos == "learned" else 0
        return self.n_layers * per_layer + emb + pos


PRESETS = {
    "70m": DecoderConfig(d_model=512, n_layers=16, n_heads=8, d_ff=2048, max_seq=256),
    "110m": DecoderConfig(d_model=768, n_layers=12, n_heads=12, d_ff=3072, max_seq=256),
    "1.3b": DecoderConfig(d_model=2048, n_layers=24, n_heads=16, d_ff=8192, max_seq=2048, act="swiglu",
                          norm="rmsnorm", pos="rope", tied=False),
    "tiny": DecoderConfig(vocab=512, d_model=128, n_layers=2, n_heads=4, d_ff=512, max_seq=64),
}


# Residual gradients are added inside the norm-backward kernel (one launch less per norm in backward:
# 6.63 -> 6.38 ms per step of the 70M decoder on one GPU); MCCL_FUSE_RESIDUAL_GRAD=0 switches it off.
_FUSE_RESIDUAL_GRAD = os.environ.get("MCCL_FUSE_RESIDUAL_GRAD", "1") != "0"


_rope_cache: dict = {}


def _rope_tables(seq: int, dim: int, device, base: float = 10000.0):
    """cos / sin of position x frequency, fp32 [seq, dim / 2].  The last few tables are kept: they depend on nothing but the
    arguments, and making them takes ten small kernels.  (Not during a graph capture: what is made there is only valid
    once the graph has run.)"""
    key = (seq, dim, str(device), base)
    tables = _rope_cache.get(key)
    if tables is not None:
        return tables
    inv = 1.0 / (base ** (torch.arange(0, dim, 2, device=device, dtype=torch.float32) / dim))
    t = torch.arange(seq, device=device, dtype=torch.float32)
    f = torch.outer(t, inv)
    tables = f.cos(), f.sin()
    if not (torch.is_inference_mode_enabled() or (f.is_cuda and torch.cuda.is_current_stream_capturing())):
        if f.is_cuda:
            torch.cuda.current_stream(f.device).synchronize()   # any stream may use them from now on
        while len(_rope_cache) >= 16:
            _rope_cache.pop(next(iter(_rope_cache)))
        _rope_cache[key] = tables
    return tables


def apply_rope(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    """x: [B, H, S, D]; rotates pairs (even, odd)."""
    x1, x2 = x[..., 0::2], x[..., 1::2]
    c, s = cos[None, None, : x.shape[2]], sin[None, None, : x.shape[2]]
    out = torch.stack((x1 * c - x2 * s, x1 * s + x2 * c), dim=-1)
    return out.flatten(-2).to(x.dtype)


# What applies to every module of the process (torch.nn.modules.module.register_module_forward_hook and friends).
_GLOBAL_HOOKS = tuple(getattr(nn.modules.module, f"_global_{kind}_hooks") for kind in ("forward", "forward_pre", "backward", "backward_pre"))


def _stock(m: nn.Module) -> bool:
    """Whether a native call may stand in for m: a module of this file, or of a class derived from one that leaves its
    methods alone."""
    return type(m).__call__ is nn.Module.__call__ and any(
        isinstance(m, cls) and all(getattr(type(m), name) is f for name, f in methods.items()) for cls, methods in _STOCK.items())


def _untouched(m: nn.Module) -> bool:
    """Whether a native call may stand in for this projection, and nobody wants to see the module's own calls.  (Host time counts
    here: twice per layer in loops that run operator by operator.)"""
    t = type(m)
    return (t.forward is _LINEAR_FORWARD and t.__call__ is _MODULE_CALL and "forward" not in m.__dict__ and not any(_GLOBAL_HOOKS)
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks))


class _Structure:
    """The parameters of some of a module's children, collected once, and whether the tree is still what it was: modules of this
    file whose methods nobody replaced, no module or parameter exchanged, no hook registered, nothing but plain fp32
    parameters.  (Walking the modules again takes longer than launching a small model's kernels.)"""

    def __init__(self, root: nn.Module, children):
        # the root itself is not among them: it keeps this object
        self.modules = list(dict.fromkeys(m for c in children if c is not None for m in c.modules()))
        self.types = [type(m) for m in self.modules]
        self.own = [m.__dict__ for m in self.modules]
        self.eps = [m.eps for m in self.modules if isinstance(m, Norm)]
        self.norms = [m.__dict__ for m in self.modules if isinstance(m, Norm)]
        self.dicts = [d for m in (root, *self.modules) for d in (m._modules, m._parameters) if d]
        self.values = [v for d in self.dicts for v in d.values()]
        self.sizes = [len(d) for d in self.dicts]
        self.hooks = [d for m in (root, *self.modules) for d in (m._forward_hooks, m._forward_pre_hooks, m._backward_hooks, m._backward_pre_hooks)]
        self.params = list(dict.fromkeys(p for m in self.modules for p in m._parameters.values() if p is not None))
        self.plain = (bool(self.params) and all(type(p) is nn.Parameter and p.dtype == torch.float32 and p.is_contiguous() for p in self.params)
                      and all(_stock(m) for m in self.modules) and len(set(self.eps)) <= 1)
        self.device = self.params[0].device if self.params else None
        self.layers = None   # the layers' parameters in order, once somebody has asked for them (False: not applicable)

    def __reduce__(self):
        return type(None), ()   # a copied or stored model collects its own

    def intact(self) -> bool:
        # (maps over built-in functions: half the time of comprehensions)
        return (self.plain and not any(self.hooks) and not any(_GLOBAL_HOOKS)
                and list(map(len, self.dicts)) == self.sizes
                and all(map(operator.is_, itertools.chain.from_iterable(map(dict.values, self.dicts)), self.values))
                and list(map(type, self.modules)) == self.types
                and not any(map(dict.__contains__, self.own, itertools.repeat("forward")))
                and list(map(operator.itemgetter("eps"), self.norms)) == self.eps
                and all([getattr(cls, name) is f for cls, name, f in _STOCK_METHODS]))


def _structure(module: nn.Module, device, children):
    """The module's cached `_Structure` of these children when it can be used on `device`, else None."""
    s = module.__dict__.get("_structure_cache")
    if s is None or s.device != device or not s.intact():
        s = _Structure(module, children)
        module.__dict__["_structure_cache"] = s
        if s.device != device or not s.intact():
            return None
    return s


# A layer as one autograd node, and a forward without gradients as one call (MCCL_FUSE_LAYER=0: operator by operator).
_FUSE_LAYER = os.environ.get("MCCL_FUSE_LAYER", "1") != "0"


class Norm(nn.Module):
    def __init__(self, cfg: DecoderConfig):
        super().__init__()
        self.kind, self.eps = cfg.norm, cfg.eps
        self.weight = nn.Parameter(torch.ones(cfg.d_model))
        self.bias = nn.Parameter(torch.zeros(cfg.d_model)) if cfg.norm == "layernorm" else None

    def forward(self, x: torch.Tensor, native: bool) -> torch.Tensor:
        if native:
            from .. import ops
            return ops.norm(x, self.weight, self.bias, self.eps)
        if self.kind == "layernorm":
            return F.layer_norm(x.float(), x.shape[-1:], self.weight, self.bias, self.eps).to(x.dtype)
        v = x.float()
        return (v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + self.eps) * self.weight).to(x.dtype)

    def with_residual(self, x: torch.Tensor, native: bool):
        """(norm(x), x as it should be fed to the residual connection).  The native path hands x through the
        norm operator so that backward adds the residual gradient in the norm-backward kernel
        (MCCL_FUSE_RESIDUAL_GRAD=0: x is returned untouched)."""
        if native and _FUSE_RESIDUAL_GRAD and type(self).forward is _NORM_FORWARD and "forward" not in self.__dict__:
            from .. import ops
            return ops.norm_residual(x, self.weight, self.bias, self.eps)
        return self.forward(x, native), x


class Linear(nn.Module):
    """Weight [out, in] (fp32 master); computes in bf16."""

    def __init__(self, d_in: int, d_out: int, bias: bool, std: float):
        super().__init__()
        self.weight = nn.Parameter(torch.empty(d_out, d_in).normal_(0.0, std))
        self.bias = nn.Parameter(torch.zeros(d_out)) if bias else None

    def forward(self, x: torch.Tensor, native: bool, act: str = "none", residual=None) -> torch.Tensor:
        if native:
            from .. import ops
            return ops.linear(x, self.weight, self.bias, act, residual)
        y = F.linear(x, self.weight.to(x.dtype), None if self.bias is None else self.bias.to(x.dtype))
        y = F.gelu(y) if act == "gelu" else y
        return y if residual is None else y + residual


class Block(nn.Module):
    def __init__(self, cfg: DecoderConfig):
        super().__init__()
        self.cfg = cfg
        d, std = cfg.d_model, 0.02
        out_std = 0.02 / math.sqrt(2 * cfg.n_layers)
        bias = cfg.norm == "layernorm"
        self.ln1 = Norm(cfg)
        self.qkv = Linear(d, 3 * d, bias, std)
        self.proj = Linear(d, d, bias, out_std)
        self.ln2 = Norm(cfg)
        if cfg.act == "swiglu":
            self.gate_up = Linear(d, 2 * cfg.d_ff, False, std)
        else:
            self.up = Linear(d, cfg.d_ff, bias, std)
        self.down = Linear(cfg.d_ff, d, bias, out_std)

    def _layer_params(self, x: torch.Tensor):
        """This layer's parameters in the order the fused layer takes them, or None where it does not apply."""
        cfg = self.cfg
        from .. import _C
        from ..ops.functional import native_attention_supported
        if cfg.norm != "layernorm" or cfg.act != "gelu" or not native_attention_supported(x.shape[1], cfg.head_dim):
            return None
        if not _C.decoder_layer_supported(x.shape[1], cfg.n_heads, cfg.d_model, cfg.d_ff):
            return None
        s = _structure(self, x.device, self._modules.values())
        if s is None:
            return None
        if s.layers is None:
            s.layers = self._ordered() or False
        if not s.layers or s.eps[0] != cfg.eps or not all(p.is_contiguous() for p in s.layers):
            return None
        if torch.is_grad_enabled() and not all(p.requires_grad for p in s.layers):
            return None   # frozen parameters: operator by operator
        return s.layers

    def _ordered(self):
        """This layer's parameters in the order the native calls take them, or None when they are not the ones its sizes ask for."""
        cfg = self.cfg
        D, FF, bias = cfg.d_model, cfg.d_ff, cfg.norm == "layernorm"
        swiglu = cfg.act == "swiglu"
        want = [("ln1", (D,), bias), ("qkv", (3 * D, D), bias), ("proj", (D, D), bias), ("ln2", (D,), bias)]
        want += [("gate_up", (2 * FF, D), False), ("down", (D, FF), bias)] if swiglu else [("up", (FF, D), bias), ("down", (D, FF), bias)]
        out = []
        for name, shape, with_bias in want:
            m = self._modules.get(name)
            if not isinstance(m, Norm if name.startswith("ln") else Linear):
                return None
            w, b = m._parameters.get("weight"), m._parameters.get("bias")
            if w is None or w.shape != shape or (b is None) == with_bias or (with_bias and b.shape != shape[:1]):
                return None
            out += [w, b] if with_bias else [w]
        return out

    def forward(self, x: torch.Tensor, rope, native: bool) -> torch.Tensor:
        cfg = self.cfg
        B, S, D = x.shape
        if native and rope is None and _FUSE_LAYER and x.dtype == torch.bfloat16:
            params = self._layer_params(x)
            if params is not None:
                from ..ops.native import DecoderLayerFn
                return DecoderLayerFn.apply(x if x.is_contiguous() else x.contiguous(), cfg.n_heads, cfg.eps, *params)
        h, x = self.ln1.with_residual(x, native)
        qkv = self.qkv(h, native)
        if native and rope is None:
            from .. import ops
            a = ops.causal_attention(qkv, cfg.n_heads)   # own kernels for S <= 256, head dimension <= 64
        elif native:
            from .. import ops
            a = ops.rope_attention(qkv, cfg.n_heads, *rope)
        else:
            qkv = qkv.view(B, S, 3, cfg.n_heads, cfg.head_dim)
            # unbind, not three selects: its backward is one stack instead of three zero-filled tensors and two adds
            q, k, v = (t.transpose(1, 2) for t in qkv.unbind(2))
            if rope is not None:
                q, k = apply_rope(q, *rope), apply_rope(k, *rope)
            a = F.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(B, S, D)
        x = self.proj(a, native, residual=x)
        h, x = self.ln2.with_residual(x, native)
        if cfg.act == "swiglu":
            if native:
                from .. import ops
                first, second = self.gate_up, self.down
                if _untouched(first) and _untouched(second) and first.bias is None and second.bias is None:
                    return ops.mlp_swiglu(h, first.weight, second.weight, residual=x)
                h = ops.swiglu(self.gate_up(h, native))   # not what the fused call computes, or somebody wants to see the calls
            else:
                g, u = self.gate_up(h, native).chunk(2, dim=-1)
                h = F.silu(g) * u
        elif native and _untouched(self.up) and _untouched(self.down):
            from .. import ops
            return ops.mlp_gelu(h, self.up.weight, self.up.bias, self.down.weight, self.down.bias, residual=x)
        else:
            h = self.up(h, native, act="gelu")
        return self.down(h, native, residual=x)


#: Modules that the native calls can stand for, and the methods whose work they do.
_STOCK = {cls: {name: getattr(cls, name) for name in ("forward", "with_residual") if hasattr(cls, name)}
          for cls in (Block, Norm, Linear, nn.Embedding, nn.ModuleList)}
_STOCK_METHODS = [(cls, name, f) for cls, methods in _STOCK.items() for name, f in methods.items()]
_LINEAR_FORWARD, _NORM_FORWARD, _MODULE_CALL = Linear.forward, Norm.forward, nn.Module.__call__


class Decoder(nn.Module):
    def __init__(self, cfg: DecoderConfig, native: Optional[bool] = None):
        super().__init__()
        self.cfg = cfg
        self.native = native
        self.tok = nn.Embedding(cfg.vocab, cfg.d_model)
        nn.init.normal_(self.tok.weight, 0.0, 0.02)
        self.pos = nn.Embedding(cfg.max_seq, cfg.d_model) if cfg.pos == "learned" else None
        if self.pos is not None:
            nn.init.normal_(self.pos.weight, 0.0, 0.02)
        self.blocks = nn.ModuleList(Block(cfg) for _ in range(cfg.n_layers))
        self.ln_f = Norm(cfg)
        self.head = None if cfg.tied else Linear(cfg.d_model, cfg.vocab, False, 0.02)
        if cfg.tied:
            # the embedding lookup contributes to this gradient through autograd as well
            self.tok.weight._shared_grad = True

    def _native(self, x: torch.Tensor) -> bool:
        if self.native is not None:
            return self.native and x.is_cuda
        return x.is_cuda

    def hidden(self, tokens: torch.Tensor) -> torch.Tensor:
        B, S = tokens.shape
        native = self._native(tokens)
        if native:
            from .. import ops
            x = ops.embedding(tokens, self.tok.weight, None if self.pos is None else self.pos.weight)
        else:
            x = self.tok(tokens)
            if self.pos is not None:
                x = x + self.pos.weight[:S]
            x = x.to(torch.bfloat16)
        rope = _rope_tables(S, self.cfg.head_dim, tokens.device) if self.cfg.pos == "rope" else None
        for blk in self.blocks:
            x = blk(x, rope, native)
        return self.ln_f(x, native)

    def _layers(self, device):
        """The structure with the layers' parameters in the order the native calls take them (`layers`) and those around them (`outer`), or
        None where those calls do not stand for this model: a module or a method was replaced, parameters are missing or of
        other sizes, somebody watches the calls."""
        cls = type(self)
        if cls.hidden is not Decoder.hidden or cls.head_weight is not Decoder.head_weight or "hidden" in self.__dict__ or "head_weight" in self.__dict__:
            return None
        m = self._modules
        s = _structure(self, device, (m.get("tok"), m.get("pos"), m.get("blocks"), m.get("ln_f"), m.get("head")))
        if s is None:
            return None
        if s.layers is None:
            cfg, layers = self.cfg, []
            for blk in self.blocks:
                own = blk._ordered() if isinstance(blk, Block) and blk.cfg == cfg else None
                if own is None:
                    layers = None
                    break
                layers += own
            tables = [t._parameters.get("weight") for t in (self.tok, self.pos, self.head) if t is not None]
            lnf = self.ln_f._parameters if isinstance(self.ln_f, Norm) else {}
            fits = (layers is not None and all(t is not None and t.dim() == 2 and t.shape[1] == cfg.d_model for t in tables)
                    and lnf.get("weight") is not None and lnf["weight"].numel() == cfg.d_model and (lnf.get("bias") is None) == (cfg.norm != "layernorm")
                    and getattr(self.head, "bias", None) is None and (self.pos is None) == (cfg.pos == "rope") and s.eps[0] == cfg.eps)
            s.layers = layers if fits else False
            if fits:
                tok, pos, head = self.tok.weight, None if self.pos is None else self.pos.weight, self.head_weight()
                s.outer = (tok, pos, self.ln_f.weight, self.ln_f.bias, head)
        return None if s.layers is False else s

    def _fused_gelu(self, tokens: torch.Tensor) -> bool:
        cfg = self.cfg
        from .. import _C
        from ..ops.functional import native_attention_supported
        return (cfg.pos == "learned" and cfg.norm == "layernorm" and cfg.act == "gelu" and tokens.dim() == 2 and tokens.dtype == torch.int64
                and tokens.shape[1] <= cfg.max_seq and not torch.is_autocast_enabled()
                and native_attention_supported(tokens.shape[1], cfg.head_dim)
                and _C.decoder_layer_supported(tokens.shape[1], cfg.n_heads, cfg.d_model, cfg.d_ff))

    def _loss_in_one_call(self, tokens: torch.Tensor, targets: torch.Tensor):
        """The training loss through C++ autograd nodes, or None where that does not apply (a trainer's gradient buffers, frozen
        or replaced parameters, hooks)."""
        if not self._fused_gelu(tokens) or targets.dtype != torch.int64 or targets.numel() != tokens.numel():
            return None
        s = self._layers(tokens.device)
        if s is None:
            return None
        tok, pos, lnf_w, lnf_b, head = s.outer
        if head.shape[0] % 8 or hasattr(tok, "_grad_sink") or not all(p.requires_grad for p in s.params):
            return None
        from .. import _C
        return _C.decoder_loss(tokens, targets, tok, pos, s.layers, lnf_w, lnf_b, head, self.cfg.n_heads, self.cfg.eps)

    def _forward_without_gradients(self, tokens: torch.Tensor):
        """Logits from one native call over the whole decoder, or None where it does not apply."""
        cfg = self.cfg
        from .. import _C
        rope = cfg.pos == "rope"
        s = self._layers(tokens.device)
        if s is None:
            return None
        tok, pos, lnf_w, lnf_b, head = s.outer
        if head.shape[0] % 8:
            return None
        if rope:
            if (tokens.dim() != 2 or tokens.dtype != torch.int64 or cfg.d_model % 64 or cfg.d_ff % 64
                    or cfg.norm != "rmsnorm" or cfg.act != "swiglu" or cfg.head_dim % 8 or torch.is_autocast_enabled()):
                return None
        elif not self._fused_gelu(tokens):
            return None
        layers = s.layers
        if hasattr(head, "_bf16"):   # a trainer keeps bf16 copies of the matrices up to date
            layers = [getattr(p, "_bf16", p) if p.dim() == 2 else p for p in layers]
            head = head._bf16
        tables = _rope_tables(tokens.shape[1], cfg.head_dim, tokens.device) if rope else (None, None)
        return _C.decoder_fwd(tokens, tok, pos, layers, lnf_w, lnf_b, head, cfg.n_heads, cfg.eps, *tables)

    def head_weight(self) -> torch.Tensor:
        return self.tok.weight if self.head is None else self.head.weight

    def forward(self, tokens: torch.Tensor, targets: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Returns logits [B, S, V] (bf16), or the mean next-token loss when targets are given."""
        if targets is None and not torch.is_grad_enabled() and _FUSE_LAYER and self._native(tokens):
            logits = self._forward_without_gradients(tokens)
            if logits is not None:
                return logits
        if targets is not None and torch.is_grad_enabled() and _FUSE_LAYER and self._native(tokens):
            loss = self._loss_in_one_call(tokens, targets)
            if loss is not None:
                return loss
        h = self.hidden(tokens)
        native = self._native(tokens)
        w = self.head_weight()
        if targets is None:
            return F.linear(h, w.to(h.dtype))
        if native:
            from .. import ops
            return ops.linear_cross_entropy(h.reshape(-1, h.shape[-1]), w, targets.reshape(-1))
        logits = F.linear(h, w.to(h.dtype))
        return F.cross_entropy(logits.float().view(-1, logits.shape[-1]), targets.reshape(-1))


def build_decoder(name: str, native: Optional[bool] = None, **overrides) -> Decoder:
    cfg = dataclasses.replace(PRESETS[name], **overrides)
    return Decoder(cfg, native=native)
