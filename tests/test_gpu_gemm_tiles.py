"""Every tile of the GEMM kernel at the edges of its tiles and of its k-blocks, against fp32 matmul."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).abs().max() / b.double().abs().max().clamp_min(1e-6)).item()


@pytest.fixture(params=["tile64", "tile128", "tile192", "pair256", ""])
def C(request):
    from mccl_b200 import _C
    _C.set_gemm_kernel(request.param)
    yield _C
    _C.set_gemm_kernel("")
    torch.cuda.synchronize()
    assert _C.gemm_error_flag() == 0


# one row, an edge in every dimension, several rounds of tiles per CTA, an odd number of 64-wide k-blocks
SHAPES = [(1, 8, 64), (37, 1536, 512), (129, 72, 192), (256, 256, 128), (257, 264, 320), (1000, 2056, 64), (8000, 2048, 576)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_product(C, M, N, K, a_t, b_t):
    if a_t:
        M = (M + 7) // 8 * 8
    torch.manual_seed(M + N + K)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref = a.float() @ b.float().t()
    aa, bb = (a.t().contiguous() if a_t else a), (b.t().contiguous() if b_t else b)
    d, _ = C.gemm_bf16(aa, bb, None, "none", False, None, False, a_t, b_t)
    assert _rel(d, ref) < 1e-2
    d, _ = C.gemm_bf16(aa, bb, None, "none", True, None, False, a_t, b_t)
    assert _rel(d, ref) < 1e-5 * max(1, K // 64)
    acc = torch.randn(M, N, device="cuda")
    want = acc + ref
    C.gemm_bf16(aa, bb, None, "none", True, acc, True, a_t, b_t)
    assert _rel(acc, want) < 1e-5 * max(1, K // 64)
    mul = torch.randn(M, N, device="cuda").bfloat16()
    d, _ = C.gemm_bf16(aa, bb, None, "none", False, None, False, a_t, b_t, None, mul)
    assert _rel(d, ref * mul.float()) < 1e-2


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_epilogues(C, M, N, K):
    torch.manual_seed(M * 3 + N + K)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16() * 0.1
    bias, res = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda").bfloat16()
    z = a.float() @ b.float().t() + bias
    assert _rel(C.gemm_bf16(a, b, bias)[0], z) < 1e-2
    assert _rel(C.gemm_bf16(a, b, bias, "none", False, None, False, False, False, res)[0], z + res.float()) < 1e-2
    d, saved = C.gemm_bf16(a, b, bias, "gelu")
    assert _rel(d, F.gelu(z)) < 1e-2 and _rel(saved, z) < 1e-2
    d, saved = C.gemm_bf16(a, b, bias, "gelu_d")
    zz = z.clone().requires_grad_(True)
    F.gelu(zz).sum().backward()
    assert _rel(d, F.gelu(z)) < 1e-2 and _rel(saved, zz.grad) < 1e-2


def test_long_contraction_is_split(C):
    torch.manual_seed(0)
    a, b = torch.randn(16384, 512, device="cuda").bfloat16(), torch.randn(16384, 256, device="cuda").bfloat16()
    d, _ = C.gemm_bf16(a, b, None, "none", True, None, False, True, True)
    assert _rel(d, a.float().t() @ b.float()) < 3e-5


@pytest.mark.parametrize("K", [8, 72, 1000])
def test_ragged_contraction(C, K):
    """Contractions that end inside a k-block: past the end the loads are zeros."""
    torch.manual_seed(K)
    a, b = torch.randn(K, 264, device="cuda").bfloat16(), torch.randn(K, 136, device="cuda").bfloat16()
    ref = a.float().t() @ b.float()
    assert _rel(C.gemm_bf16(a, b, None, "none", True, None, False, True, True)[0], ref) < 1e-5
    assert _rel(C.gemm_bf16(a.t().contiguous(), b, None, "none", False, None, False, False, True)[0], ref) < 1e-2
    assert _rel(C.gemm_bf16(a.t().contiguous(), b.t().contiguous())[0], ref) < 1e-2


@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (300, 200, 128), (4096, 2048, 512)])
def test_column_sums_of_the_output(C, M, N, K):
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    mul, acc = torch.randn(M, N, device="cuda").bfloat16(), torch.randn(N, device="cuda")
    want, ref = acc.clone(), (a.float() @ b.float()) * mul.float()
    d, _ = C.gemm_bf16(a, b, None, "none", False, None, False, False, True, None, mul, acc)
    assert _rel(d, ref) < 1e-2 and _rel(acc, want + ref.sum(0)) < 1e-4


@pytest.mark.parametrize("tokens,shapes", [(64, [(8, 8)]), (200, [(128, 64), (264, 128), (64, 512)]),
                                           (4096, [(512, 2048), (2048, 512), (512, 512), (1536, 512), (104, 72), (512, 128)])])
def test_group(tokens, shapes):
    from mccl_b200 import _C
    torch.manual_seed(tokens)
    pairs = [(torch.randn(tokens, n, device="cuda").bfloat16(), torch.randn(tokens, k, device="cuda").bfloat16()) for n, k in shapes]
    refs = [a.float().t() @ b.float() for a, b in pairs]
    tol = 1e-5 * max(1, tokens // 64)
    for d, r in zip(_C.gemm_group([(a, b, None) for a, b in pairs]), refs):
        assert _rel(d, r) < tol
    accs = [torch.randn_like(r) for r in refs]
    wants = [a + r for a, r in zip(accs, refs)]
    _C.gemm_group([(a, b, d) for (a, b), d in zip(pairs, accs)], True)
    for d, w in zip(accs, wants):
        assert _rel(d, w) < tol
    torch.cuda.synchronize()
    assert _C.gemm_error_flag() == 0
