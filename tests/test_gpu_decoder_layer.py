"""The fused decoder layer and the one-call forward against the same model operator by operator and on stock PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-12)).item()


def _pair(name, **changes):
    from mccl_b200.models import build_decoder
    torch.manual_seed(0)
    a = build_decoder(name, native=True, **changes).cuda()
    b = build_decoder(name, native=False, **changes).cuda()
    with torch.no_grad():
        for n, p in a.named_parameters():   # non-trivial norms and biases
            if p.dim() == 1:
                p.add_(torch.randn_like(p) * 0.1)
    b.load_state_dict(a.state_dict())
    return a, b


@pytest.mark.parametrize("name,changes,B,S", [("tiny", {}, 8, 24), ("tiny", {}, 3, 33), ("tiny", {"n_heads": 2, "max_seq": 256}, 2, 256),
                                              ("70m", {"n_layers": 2, "vocab": 1000}, 3, 200), ("110m", {"n_layers": 1, "vocab": 512}, 16, 256)])
def test_layer_gradients(name, changes, B, S):
    a, b = _pair(name, **changes)
    tok = torch.randint(0, a.cfg.vocab, (B, S + 1), device="cuda")
    la, lb = a(tok[:, :-1], tok[:, 1:]), b(tok[:, :-1], tok[:, 1:])
    assert abs(la.item() - lb.item()) < 2e-2
    la.backward()
    lb.backward()
    got = {n: p.grad.clone() for n, p in a.named_parameters()}
    for n, p in b.named_parameters():
        if "qkv.bias" in n:   # the key bias has no gradient but rounding
            D = a.cfg.d_model
            assert _rel(torch.cat([got[n][:D], got[n][2 * D:]]), torch.cat([p.grad[:D], p.grad[2 * D:]])) < 4e-2, n
        else:
            assert _rel(got[n], p.grad) < 4e-2, (n, _rel(got[n], p.grad))
    # gradients written into a trainer's buffers, added to what is there
    for p in a.parameters():
        p._grad_sink = torch.ones_like(p)
        p.grad = None
    a(tok[:, :-1], tok[:, 1:]).backward()
    for n, p in a.named_parameters():
        extra = p.grad if p.grad is not None else 0
        assert _rel(p._grad_sink - 1 + extra, got[n]) < 2e-2 or (got[n].abs().max() < 1e-3), n
    torch.cuda.synchronize()
    from mccl_b200 import _C
    assert _C.gemm_error_flag() == 0


SWIGLU = {"vocab": 512, "d_model": 256, "n_layers": 2, "n_heads": 4, "d_ff": 512, "max_seq": 512}


@pytest.mark.parametrize("name,changes,B,S", [("tiny", {}, 1, 1), ("tiny", {}, 5, 37), ("70m", {"n_layers": 2}, 2, 256), ("1.3b", SWIGLU, 2, 129),
                                              ("1.3b", {**SWIGLU, "n_heads": 2}, 1, 333)])
def test_forward_without_gradients(name, changes, B, S):
    a, b = _pair(name, **changes)
    tok = torch.randint(0, a.cfg.vocab, (B, S), device="cuda")
    calls = []
    inner = a._forward_without_gradients
    a._forward_without_gradients = lambda t: calls.append(inner(t)) or calls[-1]
    with torch.no_grad():
        got, want = a(tok), b(tok)
    assert calls and calls[0] is not None and got.shape == want.shape and got.dtype == torch.bfloat16
    assert _rel(got, want) < 2e-2


def test_changes_to_the_model_are_seen():
    """Replaced parameters, hooks, frozen parameters and optimizer steps: the fused paths step aside or use what is there now."""
    a, b = _pair("tiny")
    tok = torch.randint(0, a.cfg.vocab, (2, 16), device="cuda")

    def same():
        with torch.no_grad():
            assert _rel(a(tok), b(tok)) < 2e-2
        la, lb = a(tok, tok), b(tok, tok)
        assert abs(la.item() - lb.item()) < 2e-2
    same()
    with torch.no_grad():
        for m in (a, b):
            m.blocks[0].up.weight.mul_(-3.0)
    same()
    w = torch.randn_like(a.blocks[1].down.weight)
    for m in (a, b):
        m.blocks[1].down.weight = torch.nn.Parameter(w.clone())
    same()
    seen = []
    a.blocks[0].qkv.register_forward_hook(lambda *_: seen.append(1))
    same()
    assert len(seen) == 2
    a.blocks[1].proj.bias.requires_grad_(False)
    a(tok, tok).backward()
    assert a.blocks[1].proj.bias.grad is None and a.blocks[1].up.bias.grad is not None


@pytest.mark.parametrize("rows,dim,layernorm", [(1, 8, True), (37, 128, True), (1000, 512, True), (4096, 768, True), (333, 1024, True),
                                                (500, 264, False), (777, 2048, False), (600, 1024, False)])
def test_norm_backward_in_one_pass(rows, dim, layernorm):
    from mccl_b200 import _C
    torch.manual_seed(rows)
    x, dy, res = (torch.randn(rows, dim, device="cuda").bfloat16() for _ in range(3))
    w, b = torch.randn(dim, device="cuda"), torch.randn(dim, device="cuda") if layernorm else None
    y, mean, rstd = _C.norm_fwd(x, w, b, 1e-5)
    dx, dw, db = _C.norm_bwd(dy, x, w, mean, rstd, layernorm, None, None, False, res)
    gw, gb = torch.ones(dim, device="cuda"), torch.ones(dim, device="cuda")
    dx1, _, _ = _C.norm_bwd(dy, x, w, mean, rstd, layernorm, gw, gb if layernorm else None, True, res)
    assert _rel(dx1, dx) < 5e-3 and _rel(gw - 1, dw) < 1e-4
    if layernorm:
        assert _rel(gb - 1, db) < 1e-4


@pytest.mark.parametrize("kernel", ["persistent", "tile64", "tile192", "pair256"])
def test_layer_on_a_chosen_kernel(kernel):
    """What the chosen kernel does not do (ragged contractions, column sums, GELU without its second output, products times a scalar)
    goes to one that does."""
    from mccl_b200 import _C
    a, b = _pair("tiny")
    tok = torch.randint(0, a.cfg.vocab, (3, 34), device="cuda")
    try:
        for cap in (0, 1):
            _C.set_gemm_kernel(kernel)
            _C.set_gemm_cta_limit(cap)
            with torch.no_grad():
                assert _rel(a(tok), b(tok)) < 2e-2
            a.zero_grad(set_to_none=True)
            b.zero_grad(set_to_none=True)
            a(tok[:, :-1], tok[:, 1:]).backward()
            b(tok[:, :-1], tok[:, 1:]).backward()
            for (n, p), (_, q) in zip(a.named_parameters(), b.named_parameters()):
                if "qkv.bias" not in n:
                    assert _rel(p.grad, q.grad) < 4e-2, n
    finally:
        _C.set_gemm_kernel("")
        _C.set_gemm_cta_limit(0)
    assert _C.gemm_error_flag() == 0


def test_cast_many():
    from mccl_b200 import _C
    ts = [torch.randn(n, device="cuda") for n in (1, 7, 8192, 8193, 100_001)] + [torch.randn(130, 70, device="cuda") for _ in range(150)]
    for t, c in zip(ts, _C.cast_many(ts)):
        assert torch.equal(c, t.bfloat16())


@pytest.mark.parametrize("n", [1, 3, 192, 1027, 16384, 100_001])
def test_mean(n):
    from mccl_b200 import _C
    x = torch.randn(n + 1, device="cuda") + 3
    for t in (x[:n].clone(), x[1:]):   # the second does not start on 16 bytes
        assert torch.allclose(_C.mean_f32(t), t.double().mean().float(), rtol=1e-6)


@pytest.mark.parametrize("name,changes,B,S,sums", [("70m", {"n_layers": 1, "vocab": 1000}, 1, 1, True), ("70m", {"n_layers": 3, "vocab": 1000}, 1, 37, True),
                                                   ("110m", {"n_layers": 2, "vocab": 1000}, 4, 32, True), ("110m", {"n_layers": 2, "vocab": 1000}, 1, 129, False),
                                                   ("1.3b", {**SWIGLU, "d_ff": 1088}, 1, 100, True), ("1.3b", {**SWIGLU, "d_model": 2048, "n_heads": 16, "d_ff": 2112}, 2, 3, True)])
def test_few_tokens(name, changes, B, S, sums):
    """The down projections of a short forward are fp32 sums that the next norm finishes."""
    from mccl_b200 import _C
    a, b = _pair(name, **changes)
    tok = torch.randint(0, a.cfg.vocab, (B, S), device="cuda")

    def count():
        return sum(n for k, n in _C.launch_counts().items() if "norm_sum_kernel" in k)
    before = count()
    with torch.no_grad():
        got, want = a(tok), b(tok)
    assert count() - before == (a.cfg.n_layers if sums else 0)
    assert _rel(got, want) < 2e-2
    assert _C.gemm_error_flag() == 0
