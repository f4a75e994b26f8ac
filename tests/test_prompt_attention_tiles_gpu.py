"""The tcgen05 prompt attention over every small number of key tiles, with a maximum that moves in each of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 6, 9])
@pytest.mark.parametrize("rest", [1, 63, 64])
def test_a_rescale_in_every_tile(tiles, rest):
    """The rings of key and value tiles hold four, the score buffers two, and behind the last tile no scores say that a weighted
    sum is done: keys that grow from tile to tile make every row scale its sums anew in every tile, the last included.  P and the
    results are rounded to bfloat16: three half units of 2^-8 of the largest value."""
    from reinfer_b200 import ops
    QH, KH, d, page, n_new = 8, 2, 128, 16, 70
    L = 64 * (tiles - 1) + rest
    T = min(L, n_new)
    gen = torch.Generator(device=DEV).manual_seed(tiles)
    pages = -(-L // page)
    cache = torch.randn(pages, 2, KH, page, d, generator=gen, device=DEV).to(torch.bfloat16)
    strength = (torch.arange(pages * page, device=DEV) // 64 + 1).float().view(pages, 1, page)
    cache[:, 0, :, :, 3] = (12.0 * strength).to(torch.bfloat16)
    q = torch.randn(T, QH, d, generator=gen, device=DEV).to(torch.bfloat16)
    q[:, :, 3] = 20.0
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    bt, out, ref = as_int([list(range(pages))]), torch.full_like(q, float("nan")), torch.empty_like(q)
    ops.paged_attention_ref(q, cache, bt, as_int([0] * T), as_int(list(range(L - T, L))), ref, QH, KH, d, page, 0, d ** -0.5)
    for _ in range(3):
        ops.fa_prefill_tc(q, cache, bt, as_int([0, T]), as_int([L]), out, 0, 1, [T], QH, KH, d, page, 0, d ** -0.5)
        assert ops.kernel_error() == 0
        assert (out.float() - ref.float()).abs().max().item() <= 3 * 2.0 ** -9 * cache[:, 1].float().abs().max().item()
