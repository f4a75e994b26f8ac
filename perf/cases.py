"""The work that this engine's speed is measured on: batches of requests replayed through `Engine.step`.

A case is a model, a number of requests that arrive together, the range of their prompts' lengths and the number of tokens
that each of them generates.  One pass is what a serving program does with them: prompts are cut under a budget of tokens a
step and run beside the other requests' single tokens, every request leaves when it has its tokens, and the next pass begins
on an empty cache.  The generated tokens are given, as `bin/trace_run` replays them, so that a pass does the same work
whatever its logits are, and the logits at every place where a token would be drawn are its outputs.

A serving program loads one model and sees request after request: `prepare` keeps the engine of the model it was last asked
for, with fixed random weights, and makes new token ids from the seed.
"""
import functools
import math
import zlib

import numpy as np
import torch

BUDGET = 2048                # tokens a step, as LLM's default
POOL = 49152                 # tokens the cache holds
SLOTS = 64                   # requests at once, as LLM's default

# The three full-size Qwen3 shapes of reinfer_b200/shapes (hidden size, query heads, feed-forward, layers, tied output
# matrix; 8 key/value heads of 128 and a vocabulary of 151,936 in all), fewer layers where the name says so, and two designs
# at the layer sizes of `bench.py --design` (width 2,048, 16 heads, feed-forward 8,192, 6 layer runs).
QWEN3 = {"qwen3-4b": (2560, 32, 9728, 36, True), "qwen3-8b": (4096, 32, 12288, 36, False),
         "qwen3-32b-8-layers": (5120, 64, 25600, 8, False), "qwen3-4b-4-layers": (2560, 32, 9728, 4, True)}


def _case(name, model, requests, shortest, longest, new, dtype="bfloat16", page=16):
    return {"name": name, "model": model, "dtype": dtype, "page": page, "requests": requests, "shortest": shortest,
            "longest": longest, "new": new}


def listed():
    return [
        # one user's chat turn: a short prompt, then one token after the other - the smallest steps there are
        _case("one-chat", "qwen3-8b", 1, 117, 117, 24),
        # a few users with prompts of ordinary, unequal lengths
        _case("few-chats", "qwen3-8b", 8, 200, 1500, 24),
        # as many requests as fit, all short: wide decode steps
        _case("many-chats", "qwen3-4b", 64, 16, 256, 16, page=64),
        # a prompt of 2,048 tokens up to its first token
        _case("one-prompt", "qwen3-8b", 1, 2048, 2048, 1),
        # one long document in portions, and the beginning of an answer to it
        _case("document", "qwen3-4b", 1, 15877, 15877, 4, page=64),
        # requests of very different lengths: most steps hold prompt portions beside decoded tokens
        _case("mixed", "qwen3-4b", 16, 128, 2048, 24),
        # the widest layers, and contexts of a few thousand tokens in every decode step
        _case("wide-layers", "qwen3-32b-8-layers", 6, 1800, 3600, 16),
        # the 32-bit path, as a trace is replayed for comparison
        _case("float32", "qwen3-4b-4-layers", 4, 40, 300, 8, dtype="float32", page=64),
        # recurrent mixers and chunked attention: prompts, and short chats
        _case("recurrent-prompts", "silutar", 3, 400, 1200, 1),
        _case("recurrent-chats", "silutar", 8, 20, 100, 32, page=64),
        # latent attention, a recurrence with a token shift and mixtures of experts: prompts, and short chats
        _case("experts-prompts", "kibatar", 3, 400, 1200, 1),
        _case("experts-chats", "kibatar", 8, 20, 100, 32, page=64),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["qwen3-4b", "qwen3-4b", "qwen3-8b", "qwen3-8b", "qwen3-32b-8-layers", "qwen3-4b-4-layers", "silutar", "kibatar"])
    small = model == "qwen3-4b-4-layers"
    requests = log(1, 8 if small else 64)
    tokens = log(8 * requests, min(1200 if small else 8192 if model in ("silutar", "kibatar") else 16384, 4096 * requests))
    mean = max(8, tokens // requests)
    spread = rng.uniform(1.0, 3.0)
    longest = min(4095, int(mean * 2 * spread / (1 + spread)))
    return {"model": model, "dtype": "float32" if small else "bfloat16", "page": rng.choice([16, 64]), "requests": requests,
            "shortest": max(1, int(longest / spread)), "longest": longest, "new": rng.randint(1, 12 if small else 24)}


# ---------------------------------------------------------------------------------------------- models
def _raw(model):
    """config.json of the model."""
    if model in QWEN3:
        hidden, heads, ff, layers, tied = QWEN3[model]
        return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "head_dim": 128, "vocab_size": 151936, "rope_theta": 1e6,
                "rms_norm_eps": 1e-6, "max_position_embeddings": 40960, "num_hidden_layers": layers, "hidden_size": hidden,
                "num_attention_heads": heads, "num_key_value_heads": 8, "intermediate_size": ff, "tie_word_embeddings": tied}
    if model == "silutar":
        parallel = {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4, "mask": {"size": 1024}, "scale": 128 ** -0.5},
                    "right": {"heads": 16, "dim": 64, "decay_rank": 128}, "left_scale": 0.5, "right_scale": 0.5}
        delta = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 128, "gate_rank": 128}
        gla = {"heads": 16, "dim": 64, "vdim": 128, "tau": 16.0, "decay_rank": 128}
        kinds = (("parallel", parallel), ("channel_delta", delta), ("gla", gla))
        return {"architecture": "Silutar", "vocab": 32768, "width": 2048, "max_positions": 8192, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
                "layers": [{"type": kinds[i % 3][0], "mixer": kinds[i % 3][1], "mlp": {"kind": "dense", "ff": 8192}} for i in range(6)]}
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 1536, "kv_rank": 192, "scale": 192 ** -0.5,
              "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    mlp = {"kind": "moe", "expert": {"ff": 1024, "limit": 7.0}, "shared": {"ff": 2048, "limit": 7.0},
           "router": {"experts": 16, "top": 4, "scale": 1.5}}
    wkv = {"heads": 32, "dim": 64, "decay_rank": 64}
    return {"architecture": "Kibatar", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-5}, "logit_scale": 0.5,
            "embedding": {"scale": 1.0, "bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 131}},
            "loop": {"start": 1, "stop": 3, "times": 2},
            "layers": [{"type": "wkv" if i % 2 else "latent_attention", "mixer": wkv if i % 2 else latent, "mlp": mlp} for i in range(4)]}


def _tensors(model):
    """(name, shape, mean, standard deviation) of every tensor: matrices N(0, 0.02), norms' weights 1 + N(0, 0.05), wider where a
    decay, a bias, a tap or a router needs a spread of values to act on.  As in a trained model the stream of a token is not
    small beside what one layer adds to it: embeddings are wide, and the matrices (or the scales per channel) behind a sublayer
    are narrowed by the root of their number."""
    raw, out = _raw(model), []
    behind = 0.02 / math.sqrt(2 * (raw["num_hidden_layers"] if model in QWEN3 else len(raw["layers"])))

    def mat(name, *shape, std=0.02):
        out.append((name, shape, 0.0, std))

    def norm(name, *shape):
        out.append((name, shape, 1.0, 0.05))

    if model in QWEN3:
        h, ff, d, V = raw["hidden_size"], raw["intermediate_size"], 128, raw["vocab_size"]
        mat("model.embed_tokens.weight", V, h, std=1.0)
        for i in range(raw["num_hidden_layers"]):
            p = f"model.layers.{i}."
            a, f = p + "self_attn.", p + "mlp."
            norm(p + "input_layernorm.weight", h)
            mat(a + "q_proj.weight", raw["num_attention_heads"] * d, h)
            mat(a + "k_proj.weight", 8 * d, h)
            mat(a + "v_proj.weight", 8 * d, h)
            mat(a + "o_proj.weight", h, raw["num_attention_heads"] * d, std=behind)
            norm(a + "q_norm.weight", d)
            norm(a + "k_norm.weight", d)
            norm(p + "post_attention_layernorm.weight", h)
            mat(f + "gate_proj.weight", ff, h)
            mat(f + "up_proj.weight", ff, h)
            mat(f + "down_proj.weight", h, ff, std=behind)
        norm("model.norm.weight", h)
        if not raw["tie_word_embeddings"]:
            mat("lm_head.weight", V, h)
        return out
    h, V = raw["width"], raw["vocab"]
    if model == "silutar":
        def dyt(name):
            norm(name, h)
            mat(name + ".b", h, std=0.05)
            norm(name + ".alpha")

        mat("embed", V, h, std=0.2)
        mat("pos", raw["max_positions"], h)
        for i, l in enumerate(raw["layers"]):
            p, x, m = f"l{i}.", f"l{i}.mix.", l["mixer"]
            dyt(p + "norm1")
            if l["type"] == "parallel":
                a, b = m["left"], m["right"]
                for s, n in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                    mat(x + "left." + s, n, h)
                    mat(x + f"left.{s}.conv", n, a["conv"], std=0.5)
                mat(x + "left.o", h, a["heads"] * a["vdim"], std=behind)
                norm(x + "left.r1", a["heads"])
                norm(x + "left.r2", a["heads"])
                n = b["heads"] * b["dim"]
                for s in "rkvga":
                    mat(x + "right." + s, n, h)
                mat(x + "right.a.b", n, std=1.0)
                mat(x + "right.w1", b["decay_rank"], h)
                mat(x + "right.w2", n, b["decay_rank"], std=0.5)
                mat(x + "right.w0", n, std=1.0)
                norm(x + "right.norm", n)
                mat(x + "right.o", h, n, std=behind)
            elif l["type"] == "channel_delta":
                H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
                for s, n in (("q", G * dk), ("k", G * dk), ("v", H * dv)):
                    mat(x + s, n, h)
                    mat(x + s + ".conv", n, m["conv"], std=0.5)
                mat(x + "b", H, h)
                mat(x + "A_log", H, std=0.5)
                norm(x + "norm", dv)
                mat(x + "a1", m["decay_rank"], h)
                mat(x + "a2", H * dk, m["decay_rank"], std=0.5)
                mat(x + "dt_bias", H * dk, std=1.0)
                mat(x + "g1", m["gate_rank"], h)
                mat(x + "g2", H * dv, m["gate_rank"], std=0.5)
                mat(x + "o", h, H * dv, std=behind)
            else:
                H, dk, dv = m["heads"], m["dim"], m["vdim"]
                mat(x + "q", H * dk, h)
                mat(x + "k", H * dk, h)
                mat(x + "v", H * dv, h)
                mat(x + "g", H * dv, h)
                mat(x + "o", h, H * dv, std=behind)
                norm(x + "norm", dv)
                mat(x + "a1", m["decay_rank"], h)
                mat(x + "a2", H * dk, m["decay_rank"], std=0.5)
                mat(x + "a2.b", H * dk, std=1.0)
            dyt(p + "norm2")
            mat(p + "mlp.gate", l["mlp"]["ff"], h)
            mat(p + "mlp.up", l["mlp"]["ff"], h)
            mat(p + "mlp.down", h, l["mlp"]["ff"], std=behind)
        dyt("final.norm")
        return out
    mat("embed", V, h, std=1.0)
    mat("bigram", raw["embedding"]["bigram"]["buckets"] + 1, h, std=0.5)
    for i, l in enumerate(raw["layers"]):
        p, x, m, f = f"l{i}.", f"l{i}.mix.", l["mixer"], l["mlp"]
        for s in ("norm1", "norm1b", "norm2", "norm2b"):
            norm(p + s, h)
        for s in ("ls1", "ls2"):
            out.append((p + s, (h,), 10 * behind, 0.02))
        if l["type"] == "wkv":
            n = m["heads"] * m["dim"]
            for s in "rkvgw":
                mat(x + "mu." + s, h, std=0.5)
            for s in "rkvg":
                mat(x + s, n, h)
            mat(x + "w1", m["decay_rank"], h)
            mat(x + "w2", n, m["decay_rank"], std=0.5)
            mat(x + "w0", n, std=1.0)
            mat(x + "u", m["heads"], m["dim"], std=0.5)
            norm(x + "norm", n)
            mat(x + "o", h, n)
        else:
            H, dn, dr, dv = m["heads"], m["dim"], m["rot_dim"], m["vdim"]
            mat(x + "dq", m["q_rank"], h)
            norm(x + "dq.norm", m["q_rank"])
            mat(x + "uq", H * (dn + dr), m["q_rank"])
            mat(x + "uk", H * dn, m["kv_rank"])
            mat(x + "uv", H * dv, m["kv_rank"])
            mat(x + "o", h, H * dv)
            mat(x + "dkv", m["kv_rank"] + dr, h)
            norm(x + "dkv.norm", m["kv_rank"])
            mat(x + "g", H * dv, h)
            mat(x + "sink", H, std=1.0)
        mat(p + "mlp.router", f["router"]["experts"], h, std=0.1)
        mat(p + "mlp.correction", f["router"]["experts"])
        for e in [f"e{e}" for e in range(f["router"]["experts"])] + ["shared"]:
            n = f["shared" if e == "shared" else "expert"]["ff"]
            mat(p + f"mlp.{e}.gate", n, h)
            mat(p + f"mlp.{e}.up", n, h)
            mat(p + f"mlp.{e}.down", h, n)
        mat(p + "mlp.shared.sg", 1, h, std=0.1)
    mat("loop.in", h, 2 * h)
    norm("final.norm", h)
    mat("head", V, h)
    return out


def _weights(model, dtype, device):
    gen = torch.Generator(device=device).manual_seed(zlib.crc32(model.encode()))
    return {name: torch.empty(shape, dtype=getattr(torch, dtype), device=device).normal_(mean, std, generator=gen)
            for name, shape, mean, std in _tensors(model)}


@functools.lru_cache(maxsize=1)
def _engine(model, dtype, page):
    from reinfer_b200.config.registry import resolve_architecture
    from reinfer_b200.engine import Engine
    raw = _raw(model)
    arch = resolve_architecture(raw)
    config = arch.config_cls.from_dict(raw)
    return Engine(config, arch.build_spec(config), _weights(model, dtype, "cuda"), getattr(torch, dtype), page_size=page, max_tokens=POOL,
                  max_num_seqs=SLOTS, consume_state=True)


# ---------------------------------------------------------------------------------------------- the replay
def _lengths(case):
    """The prompts' lengths: spread over the range by the fractions of the golden ratio's multiples, the same for every seed."""
    lo, hi = case["shortest"], case["longest"]
    return [lo + int((hi - lo + 1) * ((k + 1) * 0.6180339887498949 % 1.0)) for k in range(case["requests"])]


def _schedule(case):
    """Steps as [(request, first token, last token + 1, whether a token is drawn behind it)]: single tokens first, then prompt
    portions in the order of arrival, BUDGET tokens in all."""
    lengths = _lengths(case)
    done, steps = [0] * len(lengths), []
    while True:
        step, room = [], BUDGET
        for r, n in enumerate(lengths):
            if n <= done[r] < n + case["new"] - 1:
                step.append((r, done[r], done[r] + 1, True))
        room -= len(step)
        for r, n in enumerate(lengths):
            if done[r] < n and room > 0:
                stop = min(n, done[r] + room)
                step.append((r, done[r], stop, stop == n))
                room -= stop - done[r]
        if not step:
            return steps
        for r, _, stop, _ in step:
            done[r] = stop
        steps.append(step)


def _tokens(case, seed):
    vocab = 151936 if case["model"] in QWEN3 else 32768
    rng = np.random.RandomState(seed % (1 << 32))
    return [rng.randint(0, vocab, n + case["new"] - 1).tolist() for n in _lengths(case)]


def prepare(case, seed):
    from reinfer_b200.engine import StepEntry
    tokens = _tokens(case, seed)
    steps = [([StepEntry(r, tokens[r][a:b], [b - a - 1] if drawn else []) for r, a, b, drawn in step],
              [r for r, _, b, _ in step if b == len(tokens[r])]) for step in _schedule(case)]
    return {"engine": _engine(case["model"], case["dtype"], case["page"]), "steps": steps}


def run(state):
    """The logits [rows, vocabulary] of every step that has any, rows in the order of the step's entries."""
    engine, outputs = state["engine"], []
    for entries, finished in state["steps"]:
        logits = engine.step(entries)
        if logits is not None:
            outputs.append(logits)
        for request in finished:
            engine.finish(request)
    return outputs


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: in every step each weight that its tokens use once (of an expert mixture the experts that so many tokens choose, on
    average), the keys, values and states that its requests read and write, and the logits.  Operations: the products and the
    attention's scores and sums over the keys that a token sees."""
    raw, isz = _raw(case["model"]), 4 if case["dtype"] == "float32" else 2
    vocab = raw["vocab_size"] if case["model"] in QWEN3 else raw["vocab"]
    shapes = {name: math.prod(shape) for name, shape, _, _ in _tensors(case["model"]) if len(shape) == 2}
    if case["model"] in QWEN3:
        runs = [f"model.layers.{i}." for i in range(raw["num_hidden_layers"])]
        hidden = raw["hidden_size"]
    else:
        order = list(range(len(raw["layers"])))
        if "loop" in raw:
            a, b, times = raw["loop"]["start"], raw["loop"]["stop"], raw["loop"]["times"]
            order = order[:a] + order[a:b] * times + order[b:]
        runs, hidden = [f"l{i}." for i in order], raw["width"]
    dense, expert, top, experts = 0, 0, 0, 0
    for p in runs:
        for name, n in shapes.items():
            if name.startswith(p):
                if ".mlp.e" in name:
                    expert += n
                else:
                    dense += n
    if case["model"] == "kibatar":
        top, experts = raw["layers"][0]["mlp"]["router"]["top"], raw["layers"][0]["mlp"]["router"]["experts"]
        dense += shapes["loop.in"] * raw["loop"]["times"]
    cached, per_key, state, chunk = 0, 0, 0, 0         # numbers cached a token, operations a key seen, bytes of state a request
    if case["model"] in QWEN3:
        cached = len(runs) * 2 * 8 * 128
        per_key = len(runs) * 4 * raw["num_attention_heads"] * 128
    for p in runs if case["model"] not in QWEN3 else ():
        l = raw["layers"][int(p[1:-1])]
        m = l["mixer"]
        if l["type"] == "latent_attention":
            cached += m["kv_rank"] + m["rot_dim"]
            per_key += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif l["type"] == "parallel":
            a, b, chunk = m["left"], m["right"], m["left"]["mask"]["size"]
            cached += a["kv_heads"] * (a["dim"] + a["vdim"])
            per_key += 2 * a["heads"] * (a["dim"] + a["vdim"])
            state += 4 * b["heads"] * b["dim"] ** 2
        else:
            state += 4 * m["heads"] * m["dim"] * m.get("vdim", m["dim"])
    moved = flops = 0.0
    for step in _schedule(case):
        n = sum(b - a for _, a, b, _ in step)
        rows = sum(drawn for _, _, _, drawn in step)
        used = experts * (1 - (1 - top / experts) ** n) / experts if experts else 0.0
        moved += isz * (dense + expert * used + n * hidden + n * cached) + 2.0 * state * len(step)
        flops += 2.0 * n * (dense + (expert * top / experts if experts else 0)) + 4.0 * n * state / 4
        if rows:
            moved += isz * vocab * hidden + 4.0 * rows * vocab
            flops += 2.0 * rows * vocab * hidden
        for _, a, b, _ in step:
            first = a // chunk * chunk if chunk else 0
            moved += isz * cached * (a - first)
            flops += per_key * sum(t + 1 - (t // chunk * chunk if chunk else 0) for t in range(a, b))
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """Four times what the engine's logits are off from `exact` (bfloat16: 0.003 to 0.0065, float32: 2.1e-6); a single value
    may move further where a rounding turns a router's choice."""
    return {"rel": 1e-5, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 0.025, "max": 0.4}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _lin(x, w):
    """x w^T; the weight's rows in parts where it is large."""
    if w.numel() < 1 << 28:
        return x @ w.to(x.dtype).t()
    return torch.cat([x @ part.to(x.dtype).t() for part in w.split(1 << 15)], dim=-1)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, positions, freqs, mag=1.0):
    """x [T, heads, d]: dimension i turns together with dimension i + n, n = len(freqs)."""
    n = len(freqs)
    ang = (positions.to(x.dtype)[:, None] * freqs)[:, None]
    c, s, u, v = torch.cos(ang) * mag, torch.sin(ang) * mag, x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], -1)


def _attend(q, k, v, scale, first=lambda i: 0 * i, bias=None, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv]: position i sees the keys from first(i) to i; 512 queries at a time."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    q = q.view(T, G, H // G, -1)
    out = []
    for a in range(0, T, 512):
        b = min(T, a + 512)
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(b, device=q.device)[None, :]
        s = torch.einsum("tgrd,sgd->grts", q[a:b], k[:b]).reshape(H, b - a, b) * scale
        if bias is not None:
            s = s + bias((i - j).clamp(min=0))
        s = s.masked_fill((j > i) | (j < first(i)), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, b - a, 1)], -1)
        s = torch.softmax(s, -1)[..., :b]
        out.append(torch.einsum("grts,sgd->tgrd", s.reshape(G, H // G, b - a, b), v[:b]).reshape(b - a, -1))
    return torch.cat(out)


class _Sequences:
    """All requests' tokens one behind the other; `each` calls a function on every request's rows, `scan` steps through all of
    them at once, padded to the longest."""

    def __init__(self, tokens, device):
        self.lengths = [len(t) for t in tokens]
        self.ids = torch.tensor([x for t in tokens for x in t], device=device)
        self.pos = torch.cat([torch.arange(n, device=device) for n in self.lengths])
        self.seq = torch.cat([torch.full((n,), r, device=device) for r, n in enumerate(self.lengths)])

    def each(self, fn, *xs):
        return torch.cat([fn(*parts) for parts in zip(*(x.split(self.lengths) for x in xs))])

    def before(self, x, steps=1):
        """The rows of so many tokens earlier, zeros before a request's first."""
        return self.each(lambda r: torch.cat([torch.zeros_like(r[:steps]), r[:-steps]])[:r.shape[0]], x)

    def scan(self, step, *xs):
        """xs [tokens, H, ...]; step(S, *one token's) -> (S, output [requests, H, dv])."""
        n = max(self.lengths)
        wide = [x.new_zeros((len(self.lengths), n) + x.shape[1:]) for x in xs]
        for w, x in zip(wide, xs):
            w[self.seq, self.pos] = x
        S, outs = None, []
        for t in range(n):
            S, o = step(S, *(w[:, t] for w in wide))
            outs.append(o)
        return torch.stack(outs, 1)[self.seq, self.pos]

    def conv(self, x, w):
        taps = w.shape[1]
        return sum((self.before(x, taps - 1 - j) if j < taps - 1 else x) * w[:, j].to(x.dtype) for j in range(taps))


def _qwen3(raw, W, s):
    eps, d, H = raw["rms_norm_eps"], 128, raw["num_attention_heads"]
    x = W["model.embed_tokens.weight"][s.ids].double()
    freqs = raw["rope_theta"] ** (-torch.arange(0, d, 2, device=x.device, dtype=x.dtype) / d)
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        w = {k[len(p):-len(".weight")]: t.double() for k, t in W.items() if k.startswith(p)}
        h = _rms(x, eps) * w["input_layernorm"]
        q, k, v = (_lin(h, w[f"self_attn.{n}_proj"]).view(x.shape[0], -1, d) for n in "qkv")
        q = _turn(_rms(q, eps) * w["self_attn.q_norm"], s.pos, freqs)
        k = _turn(_rms(k, eps) * w["self_attn.k_norm"], s.pos, freqs)
        x = x + _lin(s.each(lambda *t: _attend(*t, d ** -0.5), q, k, v), w["self_attn.o_proj"])
        h = _rms(x, eps) * w["post_attention_layernorm"]
        x = x + torch.cat([_lin(_silu(_lin(r, w["mlp.gate_proj"])) * _lin(r, w["mlp.up_proj"]), w["mlp.down_proj"]) for r in h.split(4096)])
    return _rms(x, eps) * W["model.norm.weight"].double(), lambda h: _lin(h, W.get("lm_head.weight", W["model.embed_tokens.weight"]))


def _silutar(raw, W, s):
    eps, cap = raw["norm"]["eps"], raw["logit_softcap"]

    def norm(x, name):
        return torch.tanh(W[name + ".alpha"].double() * x) * W[name].double() + W[name + ".b"].double()

    x = (W["embed"][s.ids].double() + W["pos"][s.pos].double())
    T = x.shape[0]
    for i, l in enumerate(raw["layers"]):
        p, m = f"l{i}.mix.", l["mixer"]
        w = {k[len(p):]: t.double() for k, t in W.items() if k.startswith(p)}
        h = norm(x, f"l{i}.norm1")
        if l["type"] == "gla":
            H, dk = m["heads"], m["dim"]
            q, k, v = ((_lin(h, w[n])).view(T, H, -1) for n in "qkv")
            a = (torch.sigmoid(_lin(_lin(h, w["a1"]), w["a2"]) + w["a2.b"]) ** (1.0 / m["tau"])).view(T, H, dk)

            def step(S, q, k, v, a):
                S = k[..., None] * v[..., None, :] + (0 if S is None else a[..., None] * S)
                return S, (S * q[..., None]).sum(-2)

            o = _rms(s.scan(step, q * dk ** -0.5, k, v, a), eps) * w["norm"]
            y = _lin(o.reshape(T, -1) * _silu(_lin(h, w["g"])), w["o"])
        elif l["type"] == "channel_delta":
            H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q, k, v = (_silu(s.conv(_lin(h, w[n]), w[n + ".conv"])) for n in "qkv")
            q, k = (_unit(t.view(T, G, dk)).repeat_interleave(H // G, 1) for t in (q, k))
            beta = torch.sigmoid(_lin(h, w["b"]))
            z = torch.nn.functional.softplus(_lin(_lin(h, w["a1"]), w["a2"]) + w["dt_bias"]).view(T, H, dk)
            g = torch.exp(-torch.exp(w["A_log"])[:, None] * z)

            def step(S, q, k, v, g, beta):
                S = v.new_zeros(v.shape[:2] + (dk, dv)) if S is None else g[..., None] * S
                S = S + k[..., None] * (beta[..., None] * (v - (S * k[..., None]).sum(-2)))[..., None, :]
                return S, (S * q[..., None]).sum(-2)

            o = _rms(s.scan(step, q * dk ** -0.5, k, v.view(T, H, dv), g, beta), eps) * w["norm"]
            y = _lin(o.reshape(T, -1) * torch.sigmoid(_lin(_lin(h, w["g1"]), w["g2"])), w["o"])
        else:
            a, b = m["left"], m["right"]
            q, k, v = (s.conv(_lin(h, w["left." + n]), w[f"left.{n}.conv"]).view(T, -1, a["dim"]) for n in "qkv")
            size, r1, r2 = a["mask"]["size"], w["left.r1"][:, None, None], w["left.r2"][:, None, None]
            left = s.each(lambda q, k, v: _attend(q, k, v, a["scale"], lambda i: i // size * size, lambda far: -r1 * torch.log1p(r2 * far)),
                          _rms(q, eps), _rms(k, eps), v)
            H, d = b["heads"], b["dim"]
            r, k, v, al = (t.view(T, H, d) for t in (_lin(h, w["right.r"]), _lin(h, w["right.k"]), _lin(h, w["right.v"]),
                                                     torch.sigmoid(_lin(h, w["right.a"]) + w["right.a.b"])))
            dec = torch.exp(-math.exp(-0.5) * torch.sigmoid(_lin(torch.tanh(_lin(h, w["right.w1"])), w["right.w2"]) + w["right.w0"])).view(T, H, d)

            def step(S, r, k, u, v, dec, al):
                new = k[..., None] * v[..., None, :]
                if S is not None:
                    new = new + dec[..., None] * S - (al * u)[..., None] * (S * u[..., None]).sum(-2)[..., None, :]
                return new, (new * r[..., None]).sum(-2)

            o = _rms(s.scan(step, r, k, _unit(k), v, dec, al), eps).reshape(T, -1) * w["right.norm"]
            y = m["left_scale"] * _lin(left, w["left.o"]) + m["right_scale"] * _lin(o * torch.sigmoid(_lin(h, w["right.g"])), w["right.o"])
        x = x + y
        f, h = f"l{i}.mlp.", norm(x, f"l{i}.norm2")
        x = x + _lin(_silu(_lin(h, W[f + "gate"])) * _lin(h, W[f + "up"]), W[f + "down"])
    return norm(x, "final.norm"), lambda h: cap * torch.tanh(_lin(h, W["embed"]) / cap)


def _kibatar(raw, W, s):
    eps, pair, loop = raw["norm"]["eps"], raw["embedding"]["bigram"], raw["loop"]
    prev = torch.cat([s.ids[:1], s.ids[:-1]])
    rows = torch.where(s.pos == 0, pair["buckets"], (prev * pair["mul_prev"] + s.ids * pair["mul_cur"]) % pair["buckets"])
    x0 = x = W["embed"][s.ids].double() * raw["embedding"]["scale"] + W["bigram"][rows].double()
    T = x.shape[0]
    a, b = loop["start"], loop["stop"]
    order = [(i, False) for i in range(a)] + [(i, i == a) for _ in range(loop["times"]) for i in range(a, b)]
    order += [(i, False) for i in range(b, len(raw["layers"]))]

    def expert(h, limit, p):
        g, u = _lin(h, W[p + "gate"]).clamp(max=limit), _lin(h, W[p + "up"]).clamp(-limit, limit)
        return _lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), W[p + "down"])

    for i, begins in order:
        if begins:
            x = _lin(torch.cat([x, x0], -1), W["loop.in"])
        l, p = raw["layers"][i], f"l{i}."
        m, w = l["mixer"], {k[len(p):]: t.double() for k, t in W.items() if k.startswith(p) and ".mlp.e" not in k}
        h = _rms(x, eps) * w["norm1"]
        if l["type"] == "wkv":
            H, d, before = m["heads"], m["dim"], s.before(h)
            r, k, v, g = (_lin(h + (before - h) * w["mix.mu." + n], w["mix." + n]) for n in "rkvg")
            low = torch.tanh(_lin(h + (before - h) * w["mix.mu.w"], w["mix.w1"]))
            dec = torch.exp(-torch.exp(_lin(low, w["mix.w2"]) + w["mix.w0"])).view(T, H, d)

            def step(S, r, k, v, dec):
                kv = k[..., None] * v[..., None, :]
                old = torch.zeros_like(kv) if S is None else S
                return dec[..., None] * old + kv, ((old + w["mix.u"][..., None] * kv) * r[..., None]).sum(-2)

            o = _rms(s.scan(step, *(t.view(T, H, d) for t in (r, k, v)), dec), eps)
            y = _lin(o.reshape(T, -1) * w["mix.norm"] * _silu(g), w["mix.o"])
        else:
            H, dn, rank, rot = m["heads"], m["dim"], m["kv_rank"], m["rot"]
            sc, dims = rot["scaling"], rot["dims"]

            def index(turns):
                return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))

            lo, hi = max(math.floor(index(sc["fast"])), 0), min(math.ceil(index(sc["slow"])), dims - 1)
            n = torch.arange(dims // 2, device=x.device, dtype=x.dtype)
            freqs, ramp = rot["base"] ** (-2.0 * n / dims), ((n - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
            freqs, mag = freqs / sc["factor"] * ramp + freqs * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
            q = _lin(_rms(_lin(h, w["mix.dq"]), eps) * w["mix.dq.norm"], w["mix.uq"]).view(T, H, -1)
            q = torch.cat([q[..., :dn], _turn(q[..., dn:], s.pos, freqs, mag)], -1)
            down = _lin(h, w["mix.dkv"])
            c = _rms(down[:, :rank], eps) * w["mix.dkv.norm"]
            kr = _turn(down[:, None, rank:], s.pos, freqs, mag).expand(T, H, m["rot_dim"])
            k = torch.cat([_lin(c, w["mix.uk"]).view(T, H, dn), kr], -1)
            v = _lin(c, w["mix.uv"]).view(T, H, m["vdim"])
            o = s.each(lambda q, k, v: _attend(q, k, v, m["scale"], sink=w["mix.sink"]), q, k, v)
            y = _lin(o * torch.sigmoid(_lin(h, w["mix.g"])), w["mix.o"])
        x = x + _rms(y, eps) * w["norm1b"] * w["ls1"]
        h, f = _rms(x, eps) * w["norm2"], l["mlp"]
        score = torch.softmax(_lin(h, w["mlp.router"]), -1)
        chosen = torch.topk(score + w["mlp.correction"], f["router"]["top"], -1).indices
        share = torch.zeros_like(score).scatter(1, chosen, score.gather(1, chosen)) * f["router"]["scale"]
        y = torch.sigmoid(_lin(h, w["mlp.shared.sg"])) * expert(h, f["shared"]["limit"], p + "mlp.shared.")
        for e in range(f["router"]["experts"]):
            t = share[:, e].nonzero()[:, 0]
            y[t] += share[t, e:e + 1] * expert(h[t], f["expert"]["limit"], f"{p}mlp.e{e}.")
        x = x + _rms(y, eps) * w["norm2b"] * w["ls2"]
    return _rms(x, eps) * W["final.norm"].double(), lambda h: _lin(h, W["head"]) * raw["logit_scale"]


@torch.no_grad()
def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    W = _weights(case["model"], case["dtype"], device)
    s = _Sequences(_tokens(case, seed), device)
    h, head = {"silutar": _silutar, "kibatar": _kibatar}.get(case["model"], _qwen3)(_raw(case["model"]), W, s)
    start = np.cumsum([0] + s.lengths)
    rows = [[int(start[r]) + b - 1 for r, _, b, drawn in step if drawn] for step in _schedule(case)]
    return [head(h[r]) for r in rows if r]
