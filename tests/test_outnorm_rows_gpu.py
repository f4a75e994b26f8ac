"""The output norm whose row stays in registers, at the widths where its form changes: one, two and four float4 a thread, a last
piece beyond the row, and the shared-memory form behind 4,096."""
import pytest
import torch

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("parts", [1, 3, 10])
@pytest.mark.parametrize("h", [4, 132, 1024, 1028, 2044, 2048, 2052, 4096, 4100])
def test_rows_at_the_borders(h, parts):
    from reinfer_b200 import ops
    g = torch.Generator().manual_seed(h + parts)
    T, eps, mult = 5, 1e-5, 0.4
    x, y = torch.randn(T, h, generator=g) * 3.0, torch.randn(parts, T, h, generator=g) * 0.3
    w, w1, w2 = (torch.randn(h, generator=g) * 0.1 + 1.0 for _ in range(3))
    a, src = torch.randn(T, generator=g), torch.randn(T, h, generator=g).bfloat16()
    ys = y.double().sum(0) + a.double()[:, None] * src.double()
    want = x.double() + mult * ys / torch.sqrt((ys * ys).mean(-1, keepdim=True) + eps) * w.double()
    rstd = 1.0 / torch.sqrt((want * want).mean(-1, keepdim=True) + eps)

    d = lambda t: t.to(DEV)
    streams = []
    for nxt in ("none", "next_w", "pair", "pair32"):
        s = d(x).clone()
        kw = {"next_w": {"next_w": d(w1)}, "pair": {"next_pair": (d(w1), d(w2), eps, torch.bfloat16)},
              "pair32": {"next_pair": (d(w1), d(w2), eps, torch.float32)}}.get(nxt, {})
        rounded = torch.empty(T, h, dtype=torch.bfloat16, device=DEV)
        made = ops.residual_outnorm(s, d(y), d(w), eps, mult, rounded=rounded, extra=(d(a), d(src)), **kw)
        streams.append(s)
        # parts + 1 roundings of a sum of that many terms, four more of the factor and the update: 2^-24 each of |y| or |x|
        bound = (parts + 8) * 2.0 ** -24 * (want.abs() + x.abs().double() + mult * (y.abs().double().sum(0) + (a[:, None] * src).abs()) *
                                            (want - x.double()).abs() / ys.abs().clamp_min(1e-30)) + 1e-7
        assert ((s.cpu().double() - want).abs() <= 4 * bound).all()
        assert torch.equal(rounded, s.bfloat16())
        if nxt == "next_w":
            rows, sumsq = made
            assert torch.equal(rows, (s * d(w1)).bfloat16())
            torch.testing.assert_close(sumsq.sum(1).cpu().double(), (want * want).sum(1), rtol=1e-5, atol=0)
        elif made is not None:
            for rows, wn in zip(made, (w1, w2)):
                # one rounding to bfloat16 (2^-9), a few to float (covered by it)
                torch.testing.assert_close(rows.cpu().double(), want * rstd * wn.double(), rtol=2.0 ** -8 if nxt == "pair" else 1e-5,
                                           atol=1e-5)
    assert all(torch.equal(streams[0], s) for s in streams[1:])          # what it also leaves does not change the stream
    one = d(x)[2:3].clone()                                             # nor do the rows around it
    ops.residual_outnorm(one, d(y)[:, 2:3].contiguous(), d(w), eps, mult, extra=(d(a)[2:3].contiguous(), d(src)[2:3].contiguous()))
    assert torch.equal(one, streams[0][2:3])
