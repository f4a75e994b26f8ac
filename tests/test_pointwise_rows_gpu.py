"""The 16-bit forms of the pointwise kernels that take four neighbours a lane, against 64 bits: every border of their sizes and what they
leave to the kernels that go element by element (a width or an address that is no multiple of four)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("h", [4, 6, 508, 516, 2048, 2564, 4096, 4100])
@pytest.mark.parametrize("stack,gather,shift", [(0, False, 0), (3, False, 0), (2, True, 0), (0, False, 1)])
def test_dyt(h, stack, gather, shift):
    """tanh and one product, rounded to bfloat16."""
    from reinfer_b200 import ops
    g = _gen(h)
    x = torch.randn(9, h, generator=g, device=DEV)
    w, b = (torch.randn(h + shift, generator=g, device=DEV).to(torch.bfloat16)[shift:] for _ in range(2))
    alpha = torch.tensor([0.7], device=DEV).to(torch.bfloat16)
    delta = torch.randn(stack, 9, h, generator=g, device=DEV) if stack else None
    idx = torch.tensor([8, 0, 3], dtype=torch.int32, device=DEV) if gather else None
    old, total = x.clone(), x.double() + (delta.double().sum(0) if stack else 0.0)
    rows = total[idx.long()] if gather else total
    out = torch.full(rows.shape, float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.dyt(x, delta, w, b, alpha, out, row_idx=idx)
    ref = torch.tanh(alpha.double() * rows) * w.double() + b.double()
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()
    assert torch.equal(x, old) if gather or not stack else (x.double() - total).abs().max() < 1e-5


@pytest.mark.parametrize("T,H,dv", [(1, 3, 64), (7, 5, 64), (5, 3, 128), (3, 1, 256), (4, 3, 96)])
@pytest.mark.parametrize("heads,act,shift", [(False, "silu", 0), (True, "sigmoid", 0), (True, "silu", 2)])
def test_head_norm_gate(T, H, dv, heads, act, shift):
    """Sums of dv squares in 32 bits, the result rounded to bfloat16; rows of the gate with a stride, one that does not start on 8 bytes."""
    from reinfer_b200 import ops
    g = _gen(T + dv)
    o = torch.randn(T, H, dv, generator=g, device=DEV)
    w = 1 + 0.1 * torch.randn(H * dv if heads else dv, generator=g, device=DEV)
    gate = torch.randn(T, H * dv + 16, generator=g, device=DEV).to(torch.bfloat16)[:, shift:shift + H * dv]
    out = torch.full((T, H * dv), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.head_norm_gate(o, w, gate, out, H, dv, 1e-6, act, 0.5)
    z, od = gate.double().view(T, H, dv), o.double()
    ref = od / torch.sqrt((od ** 2).mean(-1, keepdim=True) + 1e-6) * w.double().view(-1, dv) * torch.sigmoid(z) * (z if act == "silu" else 1.0) * 0.5
    assert ((out.double().view(T, H, dv) - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-6).all()


@pytest.mark.parametrize("lens", [[1], [7, 8, 9], [63, 64, 1], [65, 3], [130, 72, 17]])
@pytest.mark.parametrize("taps", [1, 2, 4, 8])
def test_short_convolution_that_reads_ahead(lens, taps):
    """Portions that end anywhere in a group of eight inputs and in a segment of 64: one chain of `taps` FMAs, rounded to bfloat16, and the
    last inputs kept for the next portion."""
    from reinfer_b200 import ops
    g, C, T = _gen(taps), 130, sum(lens)
    u = torch.randn(T, C, generator=g, device=DEV).to(torch.bfloat16)
    w = torch.randn(C, taps, generator=g, device=DEV)
    state = torch.randn(len(lens), max(taps - 1, 1), C, generator=g, device=DEV).to(torch.bfloat16).float()[:, :taps - 1].contiguous()
    before, y = state.clone(), torch.full((T, C), float("nan"), dtype=torch.bfloat16, device=DEV)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    ops.shortconv(u, w, state, y, cu, torch.arange(len(lens), dtype=torch.int32, device=DEV), len(lens), max(lens), silu=False)
    at = 0
    for e, n in enumerate(lens):
        seq = torch.cat([before[e].double(), u[at:at + n].double()])
        ref = sum(w[:, j].double() * seq[j:j + n] for j in range(taps))
        assert ((y[at:at + n].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all(), (e, n)
        assert torch.equal(state[e].double(), seq[n:])
        at += n


@pytest.mark.parametrize("T,QH,KH", [(1, 1, 1), (5, 3, 2), (33, 16, 4)])
@pytest.mark.parametrize("d,slots", [(128, True), (128, False), (96, True)])
def test_unit_heads_into_the_cache(T, QH, KH, d, slots):
    """Sums of d squares in 32 bits, rows rounded to bfloat16; a token without a slot leaves the cache alone."""
    from reinfer_b200 import ops
    g, page = _gen(T + d), 8
    x = torch.randn(T, (QH + 2 * KH) * d, generator=g, device=DEV).to(torch.bfloat16)
    slot = torch.randperm(6 * page, generator=g, device=DEV)[:T].int() if slots else None
    if slots and T > 1:
        slot[1] = -1
    cache = torch.zeros(6, 2, KH, page, d, dtype=torch.bfloat16, device=DEV)
    q = torch.full((T, QH, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.unit_heads_append(x, slot, q, cache.view(6, -1), QH, KH, d, d, page, 1e-6)
    h = x.double().view(T, QH + 2 * KH, d)
    n = h / torch.sqrt((h ** 2).mean(-1, keepdim=True) + 1e-6)
    want = torch.zeros_like(cache, dtype=torch.float64)
    for t in range(T if slots else 0):
        s = int(slot[t])
        if s >= 0:
            want[s // page, 0, :, s % page], want[s // page, 1, :, s % page] = n[t, QH:QH + KH], h[t, QH + KH:]
    close = lambda a, b: ((a.double() - b).abs() <= 2.0 ** -8 * b.abs() + 1e-6).all()
    assert close(q, n[:, :QH]) and close(cache, want)
