"""Rotary and SwiGLU kernels against the chains of PyTorch operators they replace."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).abs().max() / b.double().abs().max().clamp_min(1e-6)).item()


@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 8), (3, 37, 2, 64), (2, 333, 3, 40), (1, 1025, 16, 128)])
def test_rope_attention(B, S, H, D):
    from mccl_b200 import ops
    from mccl_b200.models.decoder import _rope_tables, apply_rope
    torch.manual_seed(S)
    qkv = torch.randn(B, S, 3 * H * D, device="cuda").bfloat16()
    cos, sin = _rope_tables(S, D, qkv.device)
    q, k, _ = (t.transpose(1, 2) for t in qkv.view(B, S, 3, H, D).unbind(2))
    from mccl_b200 import _C
    qk = _C.rope_qk_fwd(qkv.view(B, S, 3, H, D), cos, sin)
    assert torch.equal(qk[:, :, 0].transpose(1, 2), apply_rope(q, cos, sin)) and torch.equal(qk[:, :, 1].transpose(1, 2), apply_rope(k, cos, sin))
    a = qkv.clone().requires_grad_(True)
    out = ops.rope_attention(a, H, cos, sin)
    d = torch.randn_like(out)
    out.backward(d)
    r = qkv.float().requires_grad_(True)
    q, k, v = (t.transpose(1, 2) for t in r.view(B, S, 3, H, D).unbind(2))
    ref = F.scaled_dot_product_attention(apply_rope(q, cos, sin), apply_rope(k, cos, sin), v, is_causal=True).transpose(1, 2).reshape(B, S, H * D)
    ref.backward(d.float())
    assert _rel(out, ref) < 2e-2 and _rel(a.grad, r.grad) < 2e-2


@pytest.mark.parametrize("rows,f", [(1, 8), (7, 24), (333, 4096), (5000, 104)])
def test_swiglu(rows, f):
    from mccl_b200 import ops
    torch.manual_seed(rows)
    gu = (torch.randn(rows, 2 * f, device="cuda") * 3).bfloat16()
    a = gu.clone().requires_grad_(True)
    h = ops.swiglu(a)
    g, u = gu.chunk(2, dim=-1)
    assert _rel(h, F.silu(g) * u) < 1e-2
    d = torch.randn_like(h)
    h.backward(d)
    r = gu.float().requires_grad_(True)
    g, u = r.chunk(2, dim=-1)
    (F.silu(g) * u).backward(d.float())
    assert _rel(a.grad, r.grad) < 1e-2


@pytest.mark.parametrize("rows,f,k,fused", [(4096, 4096, 1024, (1, 1)), (2040, 4128, 1024, (1, 1)), (1537, 8160, 2048, (1, 1)), (37, 4096, 1024, (0, 0)), (1, 64, 64, (0, 0))])
def test_mlp_swiglu(rows, f, k, fused):
    from mccl_b200 import _C, ops
    torch.manual_seed(rows)
    x, r = (torch.randn(rows, k, device="cuda").bfloat16().requires_grad_(True) for _ in range(2))
    w1, w2 = ((torch.randn(*s, device="cuda") * s[1] ** -0.5).requires_grad_(True) for s in ((2 * f, k), (k, f)))
    x16, w16, v16 = x.detach(), w1.detach().bfloat16(), w2.detach().bfloat16()

    def separate(name, call):
        before = _C.launch_counts().get(name, 0)
        return call(), _C.launch_counts().get(name, 0) - before
    (h, gu), one = separate("swiglu_fwd_kernel", lambda: _C.gate_up_swiglu(x16, w16))
    z, _ = _C.gemm_bf16(x16, w16)
    d = torch.randn_like(x16)
    dgu, two = separate("swiglu_bwd_kernel", lambda: _C.down_swiglu_bwd(d, v16, gu))
    dh, _ = _C.gemm_bf16(d, v16, None, "none", False, None, False, False, True)
    for a, b in ((gu, z), (h, _C.swiglu_fwd(gu)), (dgu, _C.swiglu_bwd(dh, gu))):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 3e-3
    if f % 64 == 0:
        assert (1 - one, 1 - two) == fused
    ops.mlp_swiglu(x, w1, w2, residual=r).backward(d)
    xr, ar, br = (t.detach().bfloat16().float().requires_grad_(True) for t in (x, w1, w2))
    g, u = (xr @ ar.t()).chunk(2, dim=-1)
    ((F.silu(g) * u) @ br.t()).backward(d.float())
    for a, b in ((x.grad, xr.grad), (w1.grad, ar.grad), (w2.grad, br.grad), (r.grad, d)):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 1e-2
    assert _C.gemm_error_flag() == 0
