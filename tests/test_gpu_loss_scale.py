"""Gradients of a loss that is scaled or added to others before backward()."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-12)).item()


def _grads(model):
    out = {n: p.grad.clone() for n, p in model.named_parameters()}
    model.zero_grad(set_to_none=True)
    return out


SWIGLU = {"vocab": 512, "d_model": 256, "n_layers": 1, "n_heads": 4, "d_ff": 512, "max_seq": 512}


@pytest.mark.parametrize("name,changes,B,S", [("tiny", {}, 3, 33), ("tiny", {"vocab": 8192}, 8, 16), ("70m", {"n_layers": 1}, 8, 128), ("1.3b", SWIGLU, 2, 65)])
def test_scaled_and_summed_losses(name, changes, B, S):
    """The C++ nodes (GELU) and the Python one (SwiGLU); a long vocabulary's input gradient goes through partial sums."""
    from mccl_b200.models import build_decoder
    torch.manual_seed(0)
    model = build_decoder(name, **changes).cuda()
    tok = torch.randint(0, model.cfg.vocab, (2, B, S + 1), device="cuda")
    one = []
    for t in tok:
        model(t[:, :-1], t[:, 1:]).backward()
        one.append(_grads(model))
    # a power of two changes no rounding; the bound is that of sums added in another order (fp32 sums of bf16 products, bf16 gradients
    # between the layers that fall on the other side of a rounding: 2^-9 each)
    for factor in (0.25, 4096.0, -1.0):
        (model(tok[0][:, :-1], tok[0][:, 1:]) * factor).backward()
        for n, g in _grads(model).items():
            if "qkv.bias" not in n:   # the key bias has no gradient but rounding
                assert _rel(g / factor, one[0][n]) < 1e-2, (n, factor)
    (0.75 * model(tok[0][:, :-1], tok[0][:, 1:]) - 3.0 * model(tok[1][:, :-1], tok[1][:, 1:])).backward()
    for n, g in _grads(model).items():
        if "qkv.bias" not in n:
            assert _rel(g, 0.75 * one[0][n] - 3.0 * one[1][n]) < 2e-2, n
    # twice through the same graph
    loss = model(tok[0][:, :-1], tok[0][:, 1:])
    (loss * 2).backward(retain_graph=True)
    (loss * 3).backward()
    for n, g in _grads(model).items():
        if "qkv.bias" not in n:
            assert _rel(g / 5, one[0][n]) < 1e-2, n


@pytest.mark.parametrize("T,D,V", [(64, 64, 512), (200, 128, 4096), (96, 72, 1000), (7, 64, 512)])
def test_linear_cross_entropy_node(T, D, V):
    """With and without a gradient buffer, on the package's products and, where sizes do not fit them, on PyTorch's."""
    from mccl_b200 import ops
    torch.manual_seed(T)
    h = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    w = torch.nn.Parameter(torch.randn(V, D, device="cuda") * 0.05)
    y = torch.randint(0, V, (T,), device="cuda")
    hr, wr = h.detach().float().requires_grad_(), w.detach().bfloat16().float().requires_grad_()
    (torch.nn.functional.cross_entropy(hr @ wr.t(), y) * 0.3).backward()
    (ops.linear_cross_entropy(h, w, y) * 0.3).backward()
    assert _rel(h.grad, hr.grad) < 1.5e-2 and _rel(w.grad, wr.grad) < 1.5e-2
    if T % 64 == 0:
        w.grad = None
        w._grad_sink = torch.ones_like(w)
        (ops.linear_cross_entropy(h, w, y) * 0.3).backward()
        assert w.grad is None and _rel(w._grad_sink - 1, wr.grad) < 1.5e-2


@pytest.mark.parametrize("m,n,k,out_fp32,acc", [(1, 8, 8, False, False), (37, 64, 512, False, False), (136, 200, 72, True, False), (304, 264, 640, True, True),
                                                (512, 512, 8192, False, False), (1024, 4096, 512, True, True), (2048, 2048, 64, False, False)])
def test_product_times_a_device_scalar(m, n, k, out_fp32, acc):
    from mccl_b200 import _C
    torch.manual_seed(m)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(k, n, device="cuda").bfloat16()
    alpha = torch.tensor(-0.37, device="cuda")
    out = torch.ones(m, n, device="cuda") if acc else None
    d, _ = _C.gemm_bf16(a.t().contiguous() if out_fp32 else a, b, None, "none", out_fp32, out, acc, out_fp32, True, alpha=alpha)
    want = (a.double() @ b.double()) * alpha.double() + (1 if acc else 0)
    assert _rel(d, want) < (1e-5 if out_fp32 else 3e-3)
    with pytest.raises(Exception):
        _C.gemm_bf16(a, b, torch.zeros(n, device="cuda"), "none", False, None, False, False, True, alpha=alpha)
    assert _C.gemm_error_flag() == 0
