"""The recurrences over long portions of bfloat16 tokens (csrc/recurrence_chunk.cu: four tokens at a time) against the
token-by-token statement in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FORMS = [("diagonal", "sigmoid_root"), ("delta_old_state", "exp_sigmoid"), ("delta_gated_state", "exp_softplus"), ("bonus_read_first", "exp_exp")]


def _gate(kind, z, rate):
    if kind == "sigmoid_root":
        return torch.sigmoid(z) ** 0.25
    if kind == "exp_sigmoid":
        return torch.exp(-0.6 * torch.sigmoid(z))
    if kind == "exp_softplus":
        return torch.exp(-torch.exp(rate)[None, :, None] * torch.nn.functional.softplus(z))
    return torch.exp(-torch.exp(z))


def _walk(form, q, k, v, g, a, b, bonus, S):
    """q, k, g, a [n, H, dk], v [n, H, dv], b [n, H], S [H, dk, dv], all in 64 bits; one token after the other."""
    out = []
    for t in range(q.shape[0]):
        kt, vt, qt = k[t][..., None], v[t][:, None], q[t][..., None]
        if form == "diagonal":
            S = g[t][..., None] * S + kt * vt
        elif form == "bonus_read_first":
            out.append(((S + (bonus[..., None] * kt) * vt) * qt).sum(1))
            S = g[t][..., None] * S + kt * vt
            continue
        elif form == "delta_old_state":
            u = k[t] / torch.sqrt((k[t] ** 2).sum(-1, keepdim=True) + 1e-6)
            dot = (u[..., None] * S).sum(1, keepdim=True)
            S = g[t][..., None] * S - (a[t] * u)[..., None] * dot + kt * vt
        else:
            S = g[t][..., None] * S
            S = S + kt * (b[t][:, None, None] * (vt - (S * kt).sum(1, keepdim=True)))
        out.append((S * qt).sum(1))
    return torch.stack(out), S


@pytest.mark.parametrize("form,gate", FORMS)
@pytest.mark.parametrize("H,Hk,dk,dv", [(2, 2, 33, 8), (4, 2, 64, 40), (2, 1, 65, 33), (1, 1, 128, 16), (2, 2, 129, 7), (1, 1, 256, 24)])
@pytest.mark.parametrize("per_head", [False, True])
def test_chunks_of_portions_of_every_remainder(form, gate, H, Hk, dk, dv, per_head):
    """Portions that end everywhere in a pair of chunks, beside single tokens and an entry without any, in two steps over the same
    states; gates of exactly zero and within 1e-7 of one.  Tolerance: the 32-bit kernel's own over these sizes (sums of at most
    256 + 34 terms of one order, 1.2e-7 each, walked for 34 tokens: below 2e-5 of the largest output)."""
    from reinfer_b200 import ops
    if form != "delta_gated_state":
        Hk = H
        if per_head:
            pytest.skip("a gate per head belongs to the gated delta form")
    gen = torch.Generator().manual_seed(dk + dv)
    r = lambda *s: torch.randn(*s, generator=gen)
    unit, scale = form == "delta_gated_state", dk ** -0.5
    zdim = 1 if per_head else dk
    zb, ab, rate, bonus = r(H * zdim), r(H * dk), r(H) * 0.5 - 1.0, r(H * dk)
    slots = [3, 0, 5, 1, 7, 2, 6, 4]
    state = torch.full((9, H, dk, dv), float("nan"), device=DEV)
    S = {}
    for s in slots:
        state[s] = r(H, dk, dv).to(DEV) * 0.1
        S[s] = state[s].double().cpu()
    for lens in ([1, 17, 4, 0, 23, 8, 30, 2], [18, 1, 33, 12, 0, 7, 5, 34]):
        T = sum(lens)
        q, k, v = r(T, Hk * dk).bfloat16(), r(T, Hk * dk).bfloat16(), r(T, H * dv).bfloat16()
        z, a, b = r(T, H * zdim) * 2 + 1, r(T, H * dk).bfloat16(), r(T, H).bfloat16()
        shut, kept = (200.0, -30.0) if gate != "sigmoid_root" else (-600.0, 14.0)
        if not per_head:
            z.view(T, H, dk)[T // 2, :, 3] = shut
            z.view(T, H, dk)[:, :, 5] = kept
        cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
        out = torch.full((T, H, dv), float("nan"), device=DEV)
        c = lambda t: t.to(DEV)
        ops.recurrence(form, gate, c(q), c(k), c(v), c(z), c(zb), state, out, c(cu), torch.tensor(slots, dtype=torch.int32, device=DEV), len(lens),
                       H, Hk, dk, dv, gate_param={"sigmoid_root": 0.25, "exp_sigmoid": 0.6}.get(gate, 0.0), q_scale=scale, unit_qk=unit,
                       a_pre=c(a) if form == "delta_old_state" else None, a_bias=c(ab) if form == "delta_old_state" else None,
                       b_pre=c(b) if unit else None, rate=c(rate) if unit else None, max_q_len=max(lens), gate_per_head=per_head,
                       bonus=c(bonus) if form == "bonus_read_first" else None)
        assert torch.isfinite(out).all()
        for i, s in enumerate(slots):
            if not lens[i]:
                continue
            sl = slice(int(cu[i]), int(cu[i + 1]))
            qd, kd = q[sl].double().view(-1, Hk, dk), k[sl].double().view(-1, Hk, dk)
            if unit:
                qd, kd = (x / torch.sqrt((x ** 2).sum(-1, keepdim=True) + 1e-6) for x in (qd, kd))
            qd, kd = (x.repeat_interleave(H // Hk, 1) for x in (qd, kd))
            g = _gate(gate, (z[sl].double() + zb.double()).view(-1, H, zdim), rate.double()).expand(-1, H, dk)
            ref, S[s] = _walk(form, qd * scale, kd, v[sl].double().view(-1, H, dv), g, torch.sigmoid(a[sl].double() + ab.double()).view(-1, H, dk),
                              torch.sigmoid(b[sl].double()), bonus.double().view(H, dk), S[s])
            assert (out[sl].cpu().double() - ref).abs().max() < 2e-5 * ref.abs().max(), (i, lens[i])
            assert (state[s].cpu().double() - S[s]).abs().max() < 2e-5 * S[s].abs().max(), (i, lens[i])
    assert torch.isnan(state[8]).all()                          # nobody's row
