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


@pytest.mark.parametrize("rows,f,k,fused", [(4096, 4096, 1024, True), (2040, 4128, 1024, True), (1537, 8160, 2048, True), (37, 4096, 1024, False), (1, 24, 64, False)])
def test_gate_up_swiglu(rows, f, k, fused):
    from mccl_b200 import _C, ops
    torch.manual_seed(rows)
    x = torch.randn(rows, k, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(2 * f, k, device="cuda") * k ** -0.5).requires_grad_(True)
    separate = _C.launch_counts().get("swiglu_fwd_kernel", 0)
    out = ops.gate_up_swiglu(x, w)
    assert (_C.launch_counts().get("swiglu_fwd_kernel", 0) == separate) == fused
    gu = _C.gate_up_swiglu(x.detach(), w.detach().bfloat16())[1]
    z, _ = _C.gemm_bf16(x.detach(), w.detach().bfloat16())
    assert _rel(gu, z) < 1e-2 and _rel(out, _C.swiglu_fwd(gu)) < 1e-2
    assert (gu.float() - z.float()).norm() < 2e-3 * z.float().norm() and (out.float() - _C.swiglu_fwd(z).float()).norm() < 5e-3 * out.float().norm()
    d = torch.randn_like(out)
    out.backward(d)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().bfloat16().float().requires_grad_(True)
    g, u = (xr @ wr.t()).chunk(2, dim=-1)
    (F.silu(g) * u).backward(d.float())
    for a, b in ((x.grad, xr.grad), (w.grad, wr.grad)):
        assert ((a.float() - b).norm() / b.norm()).item() < 1e-2
    assert _C.gemm_error_flag() == 0
