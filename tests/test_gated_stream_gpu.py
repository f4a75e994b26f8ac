"""The gated pair over 33 to 64 tokens in the streaming kernel with a token per accumulator lane (csrc/gemm_tc.cu)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [32, 33, 47, 63, 64, 65])
@pytest.mark.parametrize("F,K", [(64, 64), (200, 72), (328, 1160), (1024, 4096)])
@pytest.mark.parametrize("scaled", [False, True])
def test_gated_pair_of_33_to_64_tokens(T, F, K, scaled):
    """Both sides of the borders, features and depth that end inside a tile; against 64 bits on the same bfloat16 operands.  The
    result is rounded to bfloat16 (2^-9 of itself), the sums are float: 1 % of the largest covers both."""
    from reinfer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(T + F)
    a = torch.randn(T, K, generator=gen, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, generator=gen, device=DEV) * K ** -0.5).to(torch.bfloat16)
    sumsq = torch.rand(T, 3, generator=gen, device=DEV) * K if scaled else None
    out = torch.full((T, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert ops.gemm_bf16_swiglu(a, w, out, row_scale=(sumsq, K, 1e-6) if scaled else None)
    gu = a.double() @ w.double().t()
    if scaled:
        gu = gu / torch.sqrt(sumsq.double().sum(1, keepdim=True) / K + 1e-6)
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    assert (out.double() - ref).abs().max() <= 0.01 * ref.abs().max()
    assert ops.kernel_error() == 0


@pytest.mark.parametrize("T", [1, 9, 16])
@pytest.mark.parametrize("F,K", [(75 * 128, 1536), (9640, 776), (148 * 128, 1032)])
@pytest.mark.parametrize("bias", [False, True])
def test_gated_pair_of_few_tokens_one_cta_an_sm(T, F, K, bias):
    """Up to 16 tokens over more than half as many tiles of features as there are SMs: the unsplit form with six stages, its first and its
    last number of tiles, with and without the epilogue's options.  Tolerance as above."""
    from reinfer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(T + F)
    a = torch.randn(T, K, generator=gen, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, generator=gen, device=DEV) * K ** -0.5).to(torch.bfloat16)
    b = torch.randn(2 * F, generator=gen, device=DEV) if bias else None
    out = torch.full((T, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert ops.gemm_bf16_swiglu(a, w, out, bias=b)
    gu = a.double() @ w.double().t() + (b.double() if bias else 0.0)
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    assert (out.double() - ref).abs().max() <= 0.01 * ref.abs().max()
    assert ops.kernel_error() == 0
