"""What repeats bit for bit: products shared out over K and what is made of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SWIGLU = {"vocab": 512, "d_model": 256, "n_layers": 2, "n_heads": 4, "d_ff": 1088, "max_seq": 512}


@pytest.mark.parametrize("name,changes,B,S", [("70m", {"n_layers": 4, "vocab": 1000}, 1, 37), ("70m", {"n_layers": 4, "vocab": 1000}, 1, 1),
                                              ("110m", {"n_layers": 2, "vocab": 1000}, 2, 64), ("1.3b", SWIGLU, 1, 100),
                                              ("1.3b", {**SWIGLU, "d_model": 2048, "n_heads": 16, "d_ff": 8192}, 1, 33)])
def test_logits_of_a_short_prompt(name, changes, B, S):
    from mccl_b200.models import build_decoder
    torch.manual_seed(0)
    model = build_decoder(name, **changes).cuda()
    tok = torch.randint(0, model.cfg.vocab, (B, S), device="cuda")
    with torch.no_grad():
        first = model(tok)
        for _ in range(20):
            assert torch.equal(model(tok), first)


@pytest.mark.parametrize("m,n,k,mn_major", [(37, 512, 4096, False), (1, 8, 4104, False), (130, 200, 5000, True), (257, 264, 4096, True), (96, 72, 32000, False), (1024, 512, 8192, True)])
def test_product_in_parts(m, n, k, mn_major):
    """Against fp64: the error of fp32 sums and one rounding to bf16 (2^-9 relative, 2-norm some half of it)."""
    from mccl_b200 import _C
    torch.manual_seed(m)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    bb = b.t().contiguous() if mn_major else b
    d, _ = _C.gemm_bf16(a, bb, b_t=mn_major)
    want = a.double() @ b.double().t()
    assert ((d.double() - want).norm() / want.norm()).item() < 2.5e-3
    for _ in range(20):
        assert torch.equal(_C.gemm_bf16(a, bb, b_t=mn_major)[0], d)
    assert _C.gemm_error_flag() == 0


@pytest.mark.parametrize("name,changes,B,S", [("tiny", {}, 8, 24), ("tiny", {"vocab": 8192}, 1, 1), ("tiny", {"n_heads": 2, "max_seq": 256}, 2, 129),
                                              ("70m", {"n_layers": 2}, 16, 256), ("110m", {"n_layers": 1, "vocab": 512}, 3, 200)])
@pytest.mark.parametrize("one_call", [True, False])
def test_vector_gradients_of_a_training_loop(monkeypatch, name, changes, B, S, one_call):
    """Biases and norms, in the loss's own call and through the layers' nodes."""
    from mccl_b200.models import build_decoder
    torch.manual_seed(0)
    model = build_decoder(name, **changes).cuda()
    if not one_call:
        monkeypatch.setattr(type(model), "_loss_in_one_call", lambda self, *a: None)
    tok = torch.randint(0, model.cfg.vocab, (B, S + 1), device="cuda")

    def grads():
        model.zero_grad(set_to_none=True)
        loss = model(tok[:, :-1], tok[:, 1:])
        loss.backward()
        return loss.detach(), {n: p.grad for n, p in model.named_parameters() if p.dim() == 1}
    l0, g0 = grads()
    assert len(g0) == 8 * model.cfg.n_layers + 2
    for _ in range(10):
        l1, g1 = grads()
        assert torch.equal(l0, l1)
        for n in g0:
            assert torch.equal(g0[n], g1[n]), n


@pytest.mark.parametrize("kernel", ["tile64", "tile128", "tile192", "pair256", "persistent"])
@pytest.mark.parametrize("m,n,k", [(37, 512, 4096), (257, 264, 4480)])
def test_product_in_parts_on_a_chosen_kernel(kernel, m, n, k):
    """The hand-chosen tile holds for products in parts, and a cap on the CTAs for how many parts there are."""
    from mccl_b200 import _C
    torch.manual_seed(m)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(k, n, device="cuda").bfloat16()
    want = a.double() @ b.double()
    try:
        for cap in (0, 20):
            _C.set_gemm_kernel(kernel)
            _C.set_gemm_cta_limit(cap)
            d, _ = _C.gemm_bf16(a, b, b_t=True)
            assert ((d.double() - want).norm() / want.norm()).item() < 2.5e-3
    finally:
        _C.set_gemm_kernel("")
        _C.set_gemm_cta_limit(0)
    assert _C.gemm_error_flag() == 0
