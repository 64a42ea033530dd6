"""Models whose modules were changed: the calls over whole layers and decoders may only stand for modules that are what they were."""
import copy
import types

import pytest
import torch
import torch.nn as nn

SWIGLU = {"vocab": 512, "d_model": 256, "n_layers": 2, "n_heads": 4, "d_ff": 512, "max_seq": 512}
MODELS = {"tiny": {"n_layers": 3}, "1.3b": SWIGLU}


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-12)).item()


def _model(name, native=None):
    from mccl_b200.models import build_decoder
    torch.manual_seed(0)
    return build_decoder(name, native=native, **MODELS[name])


class _Scaled(nn.Module):
    def forward(self, w):
        return 0.5 * w


class _Adapted(nn.Module):
    """A projection with a low-rank term beside it."""

    def __init__(self, base):
        super().__init__()
        self.base = base
        self.down = nn.Parameter(torch.randn(4, base.weight.shape[1], device=base.weight.device) * 0.1)
        self.up = nn.Parameter(torch.randn(base.weight.shape[0], 4, device=base.weight.device) * 0.1)

    def forward(self, x, native, act="none", residual=None):
        return self.base(x, native, act, residual) + (x @ self.down.t().to(x.dtype)) @ self.up.t().to(x.dtype)


def _halved(base):
    """The same parameters in a subclass with a forward of its own."""
    class Halved(type(base)):
        def forward(self, x, native, act="none", residual=None):
            return 0.5 * super().forward(x, native, act, residual)
    base.__class__ = Halved


def _parametrised(m, which):
    torch.nn.utils.parametrize.register_parametrization(getattr(m.blocks[0], which), "weight", _Scaled())


def _wrapped(m, which):
    torch.manual_seed(1)
    setattr(m.blocks[0], which, _Adapted(getattr(m.blocks[0], which)))


def _own_forward(m, which):
    lin = getattr(m.blocks[1], which)
    inner = lin.forward
    lin.forward = types.MethodType(lambda self, *a, **k: 2.0 * inner(*a, **k), lin)


def _norm_subclass(m, which):
    class Doubled(type(m.blocks[0].ln1)):
        def forward(self, x, native):
            return 2.0 * super().forward(x, native)
    m.blocks[0].ln1.__class__ = Doubled


def _other_bias(m, which):
    """A projection that has a bias where the preset has none, or none where it has one."""
    lin = getattr(m.blocks[0], which)
    torch.manual_seed(3)
    lin.bias = None if lin.bias is not None else nn.Parameter(torch.randn(lin.weight.shape[0], device=lin.weight.device))


def _resized(m, which):
    from mccl_b200.models.decoder import Linear
    blk, cfg = m.blocks[1], m.cfg
    torch.manual_seed(2)
    first = "gate_up" if cfg.act == "swiglu" else "up"
    bias, dev = blk.down.bias is not None, blk.down.weight.device
    n = cfg.d_ff // 2
    setattr(blk, first, Linear(cfg.d_model, 2 * n if cfg.act == "swiglu" else n, bias, 0.02).to(dev))
    blk.down = Linear(n, cfg.d_model, bias, 0.02).to(dev)


#: changes that no native call over a whole layer stands for
ASIDE = {"parametrised": _parametrised, "wrapped": _wrapped, "subclass": lambda m, w: _halved(getattr(m.blocks[0], w)), "own forward": _own_forward,
         "norm subclass": _norm_subclass, "bias": _other_bias, "resized": _resized,
         "eps": lambda m, w: setattr(m.blocks[1].ln1, "eps", 0.5)}
#: changes that the native calls follow
FOLLOWED = {"shared block": lambda m, w: m.blocks.__setitem__(1, m.blocks[0]), "fewer blocks": lambda m, w: setattr(m, "blocks", m.blocks[:1]),
            "swapped blocks": lambda m, w: setattr(m, "blocks", nn.ModuleList(reversed(m.blocks)))}


def _projections(name):
    return ("qkv", "proj", "down") + (("gate_up",) if name == "1.3b" else ("up",))


@pytest.mark.parametrize("name", list(MODELS))
def test_structure_is_watched(name):
    dev = torch.device("cpu")
    plain = _model(name)
    assert plain._layers(dev) is not None and plain._layers(dev).layers is plain._layers(dev).layers
    for which in _projections(name):
        for label, change in ASIDE.items():
            m = copy.deepcopy(plain)
            assert m._layers(dev) is not None
            change(m, which)
            assert m._layers(dev) is None, (label, which)
    for label, change in FOLLOWED.items():
        m = copy.deepcopy(plain)
        m._layers(dev)
        change(m, "qkv")
        found = m._layers(dev)
        want = [p for b in m.blocks for p in b._ordered()]
        assert found is not None and len(found.layers) == len(want) and all(a is b for a, b in zip(found.layers, want)), label


def test_hooks_on_every_module_are_seen():
    dev = torch.device("cpu")
    m = _model("tiny")
    assert m._layers(dev) is not None
    handle = nn.modules.module.register_module_forward_hook(lambda *_: None)
    try:
        assert m._layers(dev) is None
    finally:
        handle.remove()
    assert m._layers(dev) is not None


def test_subclass_with_its_own_hidden():
    from mccl_b200.models.decoder import Decoder

    class Other(Decoder):
        def hidden(self, tokens):
            return -super().hidden(tokens)
    m = _model("tiny")
    assert Other(m.cfg)._layers(torch.device("cpu")) is None
    assert type("Same", (Decoder,), {})(m.cfg)._layers(torch.device("cpu")) is not None


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("label", list(ASIDE) + list(FOLLOWED))
def test_changed_models_compute_what_they_say(name, label):
    """Logits, loss and gradients against the same change on stock PyTorch operators."""
    change = ASIDE.get(label) or FOLLOWED[label]
    for which in _projections(name) if label in ("parametrised", "wrapped", "subclass", "own forward", "bias") else ("qkv",):
        a, b = _model(name, True).cuda(), _model(name, False).cuda()
        tok = torch.randint(0, a.cfg.vocab, (2, 24), device="cuda")
        with torch.no_grad():
            a(tok)   # the structure is collected before the change
            for m in (a, b):
                change(m, which)
            assert _rel(a(tok), b(tok)) < 2e-2, which
        la, lb = a(tok, tok), b(tok, tok)
        assert abs(la.item() - lb.item()) < 2e-2, which
        la.backward()
        lb.backward()
        for (n, p), (_, q) in zip(a.named_parameters(), b.named_parameters()):
            if "qkv.bias" not in n:   # the key bias has no gradient but rounding
                assert _rel(p.grad, q.grad) < 4e-2, (which, n)


@pytest.mark.gpu
def test_weights_laid_out_in_another_order():
    a, b = _model("tiny", True).cuda(), _model("tiny", False).cuda()
    tok = torch.randint(0, a.cfg.vocab, (2, 24), device="cuda")
    with torch.no_grad():
        a(tok)
        w = a.blocks[0].up.weight
        w.data = w.data.t().contiguous().t()
        assert _rel(a(tok), b(tok)) < 2e-2
    la, lb = a(tok, tok), b(tok, tok)
    assert abs(la.item() - lb.item()) < 2e-2
    la.backward()
