"""The RMS norm over many rows of a prompt portion (csrc/elementwise.cu): every number of threads and pieces a row takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("h", [4, 508, 512, 516, 1540, 2560, 2564, 4100, 5120, 6148, 8192])
@pytest.mark.parametrize("wdt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("stack,shift", [(0, 0), (2, 0), (0, 1)])
def test_norm_of_many_rows(h, wdt, stack, shift):
    """Both sides of each border, with and without a stack of partial sums, and a weight that does not start on 8 bytes; 32-bit sums of
    h squares, the result rounded to bfloat16 (2^-9 of itself)."""
    from reinfer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(h)
    x = torch.randn(70, h, generator=gen, device=DEV)
    w = (1 + 0.1 * torch.randn(h + shift, generator=gen, device=DEV)).to(wdt)[shift:]
    delta = torch.randn(stack, 70, h, generator=gen, device=DEV) if stack else None
    want_x = x.double() + (delta.double().sum(0) if stack else 0.0)
    ref = want_x / torch.sqrt((want_x ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    out = torch.full((70, h), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.add_rmsnorm(x, delta, w, out, 1e-6)
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-6).all()
    assert (x.double() - want_x).abs().max() <= 1e-6 * want_x.abs().max()
