"""Attention kernels at ragged sequence lengths and head dimensions below 64, against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).abs().max() / b.double().abs().max().clamp_min(1e-6)).item()


@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 64), (2, 24, 4, 32), (3, 127, 2, 64), (2, 128, 3, 8), (2, 129, 2, 40), (8, 200, 8, 64),
                                     (2, 255, 1, 56), (2, 256, 12, 64),
                                     (65536, 2, 1, 8), (1, 3, 65537, 8), (65600, 129, 1, 8)])
def test_forward_backward_and_column_sums(B, S, H, D):
    from mccl_b200 import _C, ops
    torch.manual_seed(S * 7 + D)
    qkv = (torch.randn(B, S, 3 * H * D, device="cuda") * 1.5).bfloat16().requires_grad_(True)
    out = ops.causal_attention(qkv, H)
    d_out = (torch.randn(B, S, H * D, device="cuda") * 0.5).bfloat16()
    out.backward(d_out)
    ref_in = qkv.detach().float().requires_grad_(True)
    q, k, v = (t.transpose(1, 2) for t in ref_in.view(B, S, 3, H, D).unbind(2))
    scores = (q @ k.transpose(-1, -2)) / (D ** 0.5)
    mask = torch.ones(S, S, device="cuda", dtype=torch.bool).tril()
    ref = (scores.masked_fill(~mask, float("-inf")).softmax(-1) @ v).transpose(1, 2).reshape(B, S, H * D)
    ref.backward(d_out.float())
    assert _rel(out, ref) < 2e-2
    got, want = qkv.grad.view(B, S, 3, H, D), ref_in.grad.view(B, S, 3, H, D)
    scale = want.abs().max().clamp_min(1e-6)
    for t in range(3):   # one query: dq and dk are exactly zero, so all three are measured on one scale
        assert ((got[:, :, t].float() - want[:, :, t]).abs().max() / scale).item() < 2e-2, t
    q5 = qkv.detach().view(B, S, 3, H, D)
    o, lse = _C.attn_fwd(q5, D ** -0.5)
    sums = torch.ones(3 * H * D, device="cuda")
    d = _C.attn_bwd(q5, o, d_out, lse, D ** -0.5, sums)
    assert torch.equal(d.view_as(qkv), qkv.grad)
    assert ((sums - 1 - d.float().sum((0, 1)).view(-1)).abs().max() / d.float().abs().sum((0, 1)).max()).item() < 1e-2
    torch.cuda.synchronize()
    assert _C.gemm_error_flag() == 0


@pytest.mark.parametrize("S,D", [(257, 64), (384, 64), (128, 72), (64, 4)])
def test_other_sizes_are_refused(S, D):
    """On the host, with an error; the operator takes PyTorch's attention for them."""
    from mccl_b200 import _C
    q5 = torch.zeros(1, S, 3, 1, D, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(Exception):
        _C.attn_fwd(q5, 1.0)
    with pytest.raises(Exception):
        _C.attn_bwd(q5, torch.zeros(1, S, D, device="cuda", dtype=torch.bfloat16), torch.zeros(1, S, D, device="cuda", dtype=torch.bfloat16),
                    torch.zeros(1, 1, S, device="cuda"), 1.0)
