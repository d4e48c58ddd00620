"""GEMMs with one tile per CTA: every width, tails, layouts, epilogues; and the shapes that choose one by themselves."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, layout):
    a_mn, b_mn = layout == "mn_mn", layout != "kk"
    A = torch.randn(M, K, device="cuda").bfloat16()
    B = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    return A, B, dict(a_mn=a_mn, b_mn=b_mn), (A.t().contiguous() if a_mn else A), (B.t().contiguous() if b_mn else B)


def _close(got, want, K):
    # fp32 accumulation (error about sqrt(K) 2^-24 of a row's terms) and one rounding to bf16 (2^-9 of the value)
    scale = want.abs().max()
    return ((got.double() - want).abs().max() / scale).item() < 2 ** -8 + K * 2 ** -24


@pytest.mark.parametrize("bn", [64, 128, 192, 256])
@pytest.mark.parametrize("layout", ["kk", "k_mn", "mn_mn"])
@pytest.mark.parametrize("M,N,K", [(128, 256, 512), (72, 136, 520), (264, 8, 1000), (136, 328, 3424)])
def test_every_width(M, N, K, layout, bn):
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops import native as nv
    torch.manual_seed(M + N + K)
    A, B, kw, a, b = _operands(M, N, K, layout)
    bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    want = A.double() @ B.double().t()
    old = torch.randn(M, N, device="cuda").bfloat16()
    acc, f32 = old.clone(), torch.randn(M, N, device="cuda")
    f32_old = f32.clone()
    try:
        nv.lib().mmt_gemm_force_bn(bn)
        nv.lib().mmt_gemm_force_small(1)
        plain = F.gemm(a, b, **kw)
        full = F.gemm(a, b, bias=bias, residual=res, alpha=0.5, **kw)
        gelu = F.gemm(a, b, bias=bias, act=1, **kw)
        F.gemm(a, b, out=acc, accumulate=True, **kw)
        F.gemm(a, b, out=f32, out_f32=True, accumulate=True, **kw)
        again = F.gemm(a, b, **kw)
    finally:
        nv.lib().mmt_gemm_force_bn(0)
        nv.lib().mmt_gemm_force_small(-1)
    assert nv.get_error()[0] == 0
    assert torch.equal(plain, again)
    assert _close(plain, want, K)
    assert _close(full, 0.5 * want + bias.double() + res.double(), K)
    assert _close(gelu, torch.nn.functional.gelu(want + bias.double()), K)
    assert _close(acc, want + old.double(), K)
    assert _close(f32, want + f32_old.double(), K)


@pytest.mark.parametrize("M", [1, 64, 129, 256, 443, 1024])
@pytest.mark.parametrize("N,K", [(1280, 1280), (1280, 3424), (3840, 1280), (2048, 11008), (64, 256), (8, 64)])
def test_shapes_that_do_not_fill_the_gpu(M, N, K):
    from multimodal_training_b200.ops import functional as F
    torch.manual_seed(M + N + K)
    A, B, kw, a, b = _operands(M, N, K, "kk")
    assert _close(F.gemm(a, b), A.double() @ B.double().t(), K)


@pytest.mark.parametrize("layout", ["kk", "k_mn", "mn_mn"])
@pytest.mark.parametrize("bn", [64, 128, 192, 256])
def test_one_tile_per_cta_has_the_bits_of_the_persistent_kernel(bn, layout):
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops import native as nv
    torch.manual_seed(bn)
    A, B, kw, a, b = _operands(264, 328, 1000, layout)
    bias, res = torch.randn(328, device="cuda").bfloat16(), torch.randn(264, 328, device="cuda").bfloat16()
    got = []
    try:
        nv.lib().mmt_gemm_force_bn(bn)
        for small in (0, 1):
            nv.lib().mmt_gemm_force_small(small)
            acc = res.clone()
            F.gemm(a, b, out=acc, accumulate=True, **kw)
            got.append((F.gemm(a, b, bias=bias, residual=res, **kw), F.gemm(a, b, bias=bias, act=1, **kw), acc))
    finally:
        nv.lib().mmt_gemm_force_bn(0)
        nv.lib().mmt_gemm_force_small(-1)
    assert all(torch.equal(x, y) for x, y in zip(*got))
