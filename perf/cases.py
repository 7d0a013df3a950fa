"""The work that is timed: what a program that generates with this library has it do.

Three ways in, as programs use them: a Session's step (prompts, portions onto started sequences, decode steps;
whole models and stacks of one or two layers at a model's full widths), the mixture-of-experts part, and the
kernels' own entry points for attention over packed prompts and for the state mixers' scan. Widths are those of
the shapes the benchmark names (the Llama 3 1B, 3B and 8B shapes; the 2,048-wide layers of the other designs).
Weights are drawn as `Engine.random` draws them, token ids and activations from the case's seed.
"""
import hashlib
import math
import random

import numpy as np
import torch

# hidden, feed-forward, heads, key/value heads, head size, rotation factor, tied head
SHAPES = {
    "1b": (2048, 8192, 32, 8, 64, 32.0, True),
    "3b": (3072, 8192, 24, 8, 128, 32.0, True),
    "8b": (4096, 14336, 32, 8, 128, 8.0, False),
}
STD, NORM_STD, EPS, THETA = 0.02, 0.1, 1e-5, 500000.0


def listed():
    return [
        # One user's chat: a single sequence, a few hundred tokens in. The smallest step there is.
        dict(name="decode-1b-b1", kind="decode", shape="1b", layers=2, vocab=32768, batch=1, low=300, high=300, dtype="bfloat16"),
        # The benchmark's headline: eight requests half way to a context of 4,096, the whole model.
        dict(name="decode-1b-b8-whole", kind="decode", shape="1b", layers=16, vocab=128256, batch=8, low=2176, high=3072,
             dtype="bfloat16"),
        # A loaded server: many requests of very unequal length up to 8,000 tokens, wide layers.
        dict(name="decode-8b-b32", kind="decode", shape="8b", layers=2, vocab=32768, batch=32, low=1000, high=8000,
             dtype="bfloat16"),
        # Time to first token of one 2,048-token prompt, the whole model.
        dict(name="prompt-1b-whole", kind="prompt", shape="1b", layers=16, vocab=128256, lengths="2048", dtype="bfloat16"),
        # A batch of new requests of unequal, odd lengths that start together.
        dict(name="prompt-3b-packed", kind="prompt", shape="3b", layers=2, vocab=32768, lengths="700,1333,64,257,1999",
             dtype="bfloat16"),
        # A second turn: new text onto two conversations that are in the cache already.
        dict(name="extend-8b", kind="extend", shape="8b", layers=2, vocab=32768, held="3000,1111", lengths="400,129",
             dtype="bfloat16"),
        # The true 32-bit path, which numerical work and the parity checks use.
        dict(name="prompt-1b-f32", kind="prompt", shape="1b", layers=1, vocab=8192, lengths="333", dtype="float32"),
        # Attention alone over packed prompts, the 1B shape's heads.
        dict(name="attention-packed", kind="attention", heads=32, kv_heads=8, dim=64, window=0, lengths="3001,517,1200"),
        # Experts while eight sequences decode (the 2,048-wide layers of the expert designs).
        dict(name="moe-rows8", kind="moe", width=2048, ff=1024, experts=8, top=2, rows=8),
        # Experts of a prompt.
        dict(name="moe-prompt", kind="moe", width=2048, ff=1024, experts=8, top=2, rows=1500),
        # State mixers over a prompt: the gated delta rule, and a decay per head and token over two prompts.
        dict(name="scan-delta", kind="scan", rule="delta", heads=16, key_heads=4, dim=128, vdim=128, lengths="2048"),
        dict(name="scan-decay", kind="scan", rule="token_decay", heads=32, key_heads=1, dim=128, vdim=64, lengths="1500,777"),
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _lengths(rng, total, most):
    """Up to `most` lengths that add up to `total`."""
    count = min(rng.randint(1, most), total)
    cuts = sorted(rng.sample(range(1, total), count - 1)) if count > 1 else []
    return [b - a for a, b in zip([0] + cuts, cuts + [total])]


def _text(numbers):
    return ",".join(str(n) for n in numbers)


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "extend", "float32", "attention", "moe", "scan", "scan"])
    if kind == "decode":
        batch = _log_uniform(rng, 1, 64)
        high = _log_uniform(rng, 64, min(8000, 200000 // batch))
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), layers=rng.randint(1, 2), vocab=rng.choice([8192, 32768]),
                    batch=batch, low=max(1, int(high * rng.uniform(0.1, 1.0))), high=high, dtype="bfloat16")
    if kind == "prompt":
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), layers=rng.randint(1, 2), vocab=rng.choice([8192, 32768]),
                    lengths=_text(_lengths(rng, _log_uniform(rng, 16, 4096), 6)), dtype="bfloat16")
    if kind == "extend":
        lengths = _lengths(rng, _log_uniform(rng, 8, 1024), 4)
        lengths[0] += 1  # more than one token: a portion, not a decode step
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), layers=rng.randint(1, 2), vocab=32768,
                    held=_text(_log_uniform(rng, 16, 4000) for _ in lengths), lengths=_text(lengths), dtype="bfloat16")
    if kind == "float32":
        return dict(kind="prompt", shape="1b", layers=1, vocab=8192, lengths=_text(_lengths(rng, _log_uniform(rng, 4, 512), 3)),
                    dtype="float32")
    if kind == "attention":
        heads, kv_heads, dim = rng.choice([(32, 8, 64), (24, 8, 128), (32, 8, 128), (16, 4, 128), (8, 2, 64)])
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, dim=dim, window=rng.choice([0, 0, 0, 512, 1024]),
                    lengths=_text(_lengths(rng, _log_uniform(rng, 32, 6000), 4)))
    if kind == "moe":
        width, ff = rng.choice([(1024, 512), (2048, 1024)])
        experts, top = rng.choice([(8, 2), (8, 2), (16, 4), (32, 2)])
        return dict(kind=kind, width=width, ff=ff, experts=experts, top=top, rows=_log_uniform(rng, 1, 2048 if experts < 32 else 64))
    heads, key_heads, dim, vdim = rng.choice([(16, 4, 128, 128), (8, 8, 128, 128), (16, 16, 64, 64), (32, 1, 128, 64), (4, 2, 96, 80)])
    return dict(kind="scan", rule=rng.choice(["delta", "token_decay", "head_decay"]), heads=heads, key_heads=key_heads, dim=dim,
                vdim=vdim, lengths=_text(_lengths(rng, _log_uniform(rng, 16, 4096), 4)))


# ---------------------------------------------------------------------------- what a case consists of
def _numbers(text):
    return [int(n) for n in text.split(",")]


def _config(case):
    hidden, ff, heads, kv_heads, dim, factor, tied = SHAPES[case["shape"]]
    return dict(
        architectures=["LlamaForCausalLM"], model_type="llama", hidden_size=hidden, intermediate_size=ff,
        num_hidden_layers=case["layers"], num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim,
        vocab_size=case["vocab"], rope_theta=THETA,
        rope_scaling=dict(rope_type="llama3", factor=factor, low_freq_factor=1.0, high_freq_factor=4.0,
                          original_max_position_embeddings=8192),
        rms_norm_eps=EPS, tie_word_embeddings=tied, max_position_embeddings=131072)


def _held(case):
    """How many tokens each sequence has in the cache before the pass."""
    if case["kind"] == "decode":
        spread = random.Random("%d %d %d" % (case["batch"], case["low"], case["high"]))
        return [spread.randint(case["low"], case["high"]) for _ in range(case["batch"])]
    if case["kind"] == "extend":
        return _numbers(case["held"])
    return [0] * len(_numbers(case["lengths"]))


def _brought(case):
    return [1] * case["batch"] if case["kind"] == "decode" else _numbers(case["lengths"])


def _tokens(case, seed):
    """Every sequence's token ids: what it holds, then what the pass brings."""
    rng = np.random.default_rng(seed)
    return [rng.integers(0, case["vocab"], size=held + new).tolist() for held, new in zip(_held(case), _brought(case))]


def _randn(seed, name, *shape):
    generator = torch.Generator(device="cuda").manual_seed(int.from_bytes(
        hashlib.sha256(("%d:%s" % (seed, name)).encode()).digest()[:8], "little") >> 1)
    return torch.randn(shape, generator=generator, dtype=torch.float32, device="cuda")


def _rand(seed, name, *shape):
    return torch.special.ndtr(_randn(seed, name, *shape))


def _scan_inputs(case, seed):
    """As the mixers prepare them: unit keys, scaled unit queries, decays a little below one, steps between 0 and 1."""
    T, H, G, d, dv = sum(_numbers(case["lengths"])), case["heads"], case["key_heads"], case["dim"], case["vdim"]
    q = torch.nn.functional.normalize(_randn(seed, "q", T, G, d), dim=-1) * d ** -0.5
    k = torch.nn.functional.normalize(_randn(seed, "k", T, G, d), dim=-1)
    v = _randn(seed, "v", T, H, dv)
    rates = torch.linspace(math.log(1e-3), math.log(0.3), H, device="cuda").exp()  # slow heads to fast ones
    if case["rule"] == "delta":
        more = dict(g=torch.exp(-rates[None, :, None] * 2 * _rand(seed, "g", T, H, d)).contiguous(),
                    beta=_rand(seed, "beta", T, H).contiguous())
    elif case["rule"] == "token_decay":
        more = dict(token_decay=torch.exp(-rates[None, :] * 2 * _rand(seed, "g", T, H)).contiguous())
    else:
        more = dict(head_decay=torch.exp(-rates).contiguous())
    return q.contiguous(), k.contiguous(), v.contiguous(), more


def _moe_inputs(case, seed):
    h, f, E = case["width"], case["ff"], case["experts"]
    tensors = {"router.weight": _randn(seed, "router", E, h) * STD}
    for e in range(E):
        for name, shape in (("gate_proj", (f, h)), ("up_proj", (f, h)), ("down_proj", (h, f))):
            tensors["experts.%d.%s.weight" % (e, name)] = (_randn(seed, "%d.%s" % (e, name), *shape) * STD).to(torch.bfloat16)
    return _randn(seed, "x", case["rows"], h).to(torch.bfloat16), tensors


def _attention_inputs(case, seed):
    T = sum(_numbers(case["lengths"]))
    return tuple(_randn(seed, name, T, heads, case["dim"]).to(torch.bfloat16)
                 for name, heads in (("q", case["heads"]), ("k", case["kv_heads"]), ("v", case["kv_heads"])))


def _int32(numbers):
    return torch.tensor(numbers, dtype=torch.int32, device="cuda")


# ---------------------------------------------------------------------------- one pass
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prompt", "extend"):
        from llama_rs_metal_b200 import Engine
        from llama_rs_metal_b200.engine.batch import StepEntry
        model = Engine().random(_config(case), seed=seed, std=STD, norm_std=NORM_STD, dtype=case["dtype"])
        tokens, held, new = _tokens(case, seed), _held(case), _brought(case)
        session = model.session(context=-(-(max(len(t) for t in tokens) + 1) // 64) * 64, max_batch=len(tokens))
        state = dict(kind=kind, session=session, new=[t[n:] for t, n in zip(tokens, held)], StepEntry=StepEntry)
        if kind != "prompt":  # the conversation so far
            state["slots"] = [session.open_slot() for _ in tokens]
            for at in range(0, len(tokens), 8):
                session.step([StepEntry(slot, t[:n], ()) for slot, t, n in zip(state["slots"], tokens, held)][at:at + 8])
        if kind == "decode":  # a generation that is under way: its steps are captured
            run(state)
        return state
    if kind == "moe":
        from llama_rs_metal_b200.parts.moe import MixtureOfExperts
        from llama_rs_metal_b200.runtime import Runtime
        x, tensors = _moe_inputs(case, seed)
        moe = MixtureOfExperts(case["width"], case["ff"], case["experts"], case["top"], router_bias=False)
        moe.bind(tensors, Runtime(x.device, torch.bfloat16))
        return dict(kind=kind, x=x, moe=moe)
    lengths = _numbers(case["lengths"])
    state = dict(kind=kind, cu_seqlens=_int32(np.cumsum([0] + lengths).tolist()))
    if kind == "attention":
        state["q"], state["k"], state["v"] = _attention_inputs(case, seed)
        state["seq_of_token"] = _int32(np.repeat(np.arange(len(lengths)), lengths).tolist())
        state.update(longest=max(lengths), scale=case["dim"] ** -0.5, window=case["window"] or None)
        return state
    state["q"], state["k"], state["v"], state["more"] = _scan_inputs(case, seed)
    state["state"] = torch.zeros(len(lengths), case["heads"], case["dim"], case["vdim"], device="cuda")
    state["slots"] = _int32(list(range(len(lengths))))
    return state


def run(state):
    kind = state["kind"]
    if kind == "moe":  # as a block with a norm behind the part runs it: float32, not yet added to the stream
        return state["moe"].forward(state["x"], None, None)
    if kind in ("attention", "scan"):
        from llama_rs_metal_b200.kernels import ops
        if kind == "attention":
            return ops.attention_prefill(state["q"], state["k"], state["v"], state["cu_seqlens"], state["seq_of_token"],
                                         state["longest"], state["scale"], state["window"])
        state["state"].zero_()  # new sequences start from nothing
        out = ops.linear_state_scan(state["q"], state["k"], state["v"], state["state"], state["cu_seqlens"], state["slots"],
                                    **state["more"])
        return out, state["state"]
    session, entry = state["session"], state["StepEntry"]
    if kind == "prompt":
        slots = [session.open_slot() for _ in state["new"]]
        logits = session.step([entry(slot, t, (len(t) - 1,)) for slot, t in zip(slots, state["new"])])
        for slot in slots:
            session.close_slot(slot)
        return logits
    logits = session.step([entry(slot, t, (len(t) - 1,)) for slot, t in zip(state["slots"], state["new"])])
    for slot, t in zip(state["slots"], state["new"]):  # so that the next pass does the same work
        session.rewind([slot], len(t))
    return logits


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prompt", "extend"):
        hidden, ff, heads, kv_heads, dim, _, _ = SHAPES[case["shape"]]
        held, new, elem = _held(case), _brought(case), 4 if case["dtype"] == "float32" else 2
        layer = hidden * (heads + 2 * kv_heads) * dim + heads * dim * hidden + 3 * hidden * ff
        rows, tokens = len(new), sum(new)
        pairs = sum(n * h + n * (n + 1) // 2 for h, n in zip(held, new))
        return dict(
            bytes=(case["layers"] * (layer + 2 * hidden) + (case["vocab"] + 1 + min(tokens, case["vocab"])) * hidden) * elem
            + case["layers"] * 2 * kv_heads * dim * elem * (sum(held) + tokens) + rows * case["vocab"] * 4,
            flops=case["layers"] * (2 * layer * tokens + 4 * pairs * heads * dim) + 2 * rows * case["vocab"] * hidden)
    if kind == "moe":
        h, f, E, top, rows = case["width"], case["ff"], case["experts"], case["top"], case["rows"]
        used = E * (1.0 - (1.0 - top / E) ** rows)  # experts that somebody chose
        return dict(bytes=used * 3 * h * f * 2 + E * h * 4 + rows * h * (2 + 4), flops=rows * (top * 6 * h * f + 2 * E * h))
    lengths = _numbers(case["lengths"])
    T = sum(lengths)
    if kind == "attention":
        window = case["window"] or max(lengths)
        pairs = sum(n * (n + 1) // 2 - max(0, n - window) * (max(0, n - window) + 1) // 2 for n in lengths)
        return dict(bytes=2 * T * case["dim"] * (2 * case["heads"] + 2 * case["kv_heads"]), flops=4 * pairs * case["heads"] * case["dim"])
    H, G, d, dv = case["heads"], case["key_heads"], case["dim"], case["vdim"]
    decays = {"delta": T * H * (d + 1), "token_decay": T * H, "head_decay": H}[case["rule"]]
    return dict(bytes=4 * (2 * T * G * d + 2 * T * H * dv + decays + len(lengths) * H * d * dv),
                flops=(7 if case["rule"] == "delta" else 5) * T * H * d * dv)


def tolerance(case):
    """About four times the distance from 64 bits that was measured."""
    kind = case["kind"]
    if kind in ("decode", "prompt", "extend"):
        if case["dtype"] == "float32":
            return {"rel": 1.6e-5}                                 # 4.0e-6
        return {"rel": 7e-2 if case["layers"] > 2 else 5e-2}       # 1.8e-2 (16 layers), 0.7e-2 to 1.3e-2 (1 or 2)
    if kind == "moe":  # few rows keep float32 between the products (2.5e-7), many round to bfloat16 there (1.7e-3)
        return {"rel": 7e-3 if case["rows"] >= 64 and case["experts"] <= 4 * case["top"] else 1e-6}
    return {"rel": 8e-3 if kind == "attention" else 2e-6}          # 2.1e-3, and 1e-7 to 5.6e-7


# ---------------------------------------------------------------------------- the same in 64 bits
def _weight(case, seed, name, *shape):
    t = _randn(seed, name, *shape)
    if len(shape) == 1:
        t = t * NORM_STD + 1.0
    else:
        t.mul_(STD)
    return (t if case["dtype"] == "float32" else t.to(torch.bfloat16)).double()


def _frequencies(dim, factor):
    """Llama 3's scaled rotation: long wavelengths slowed by `factor`, a blend in between."""
    out = []
    for i in range(dim // 2):
        freq = THETA ** (-2.0 * i / dim)
        wave = 2 * math.pi / freq
        if wave > 8192 / 1.0:
            freq /= factor
        elif wave > 8192 / 4.0:
            smooth = (8192 / wave - 1.0) / (4.0 - 1.0)
            freq = (1 - smooth) * freq / factor + smooth * freq
        out.append(freq)
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _rms(x, weight):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * weight


def _attend(q, k, v, scale, window, first):
    """q [n, H, d], whose rows are positions first .. first + n - 1, over k, v [m, G, d]."""
    n, H, _ = q.shape
    group = H // k.shape[1]
    at, key = torch.arange(first, first + n, device="cuda")[:, None], torch.arange(k.shape[0], device="cuda")[None, :]
    hidden = key > at
    if window:
        hidden |= key <= at - window
    out = torch.empty(n, H, v.shape[2], dtype=torch.float64, device="cuda")
    for h in range(H):
        scores = (q[:, h] @ k[:, h // group].T * scale).masked_fill_(hidden, -math.inf)
        out[:, h] = torch.softmax(scores, -1) @ v[:, h // group]
    return out


def _exact_model(case, seed):
    hidden, ff, heads, kv_heads, dim, factor, tied = SHAPES[case["shape"]]
    embedding = _weight(case, seed, "model.embed_tokens.weight", case["vocab"], hidden)
    sequences = [embedding[torch.tensor(t, device="cuda")] for t in _tokens(case, seed)]
    freq = _frequencies(dim, factor)

    def turn(x):  # split halves
        angle = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None] * freq
        cos, sin = angle.cos()[:, None], angle.sin()[:, None]
        a, b = x[..., :dim // 2], x[..., dim // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for i in range(case["layers"]):
        at = "model.layers.%d." % i
        w = lambda name, *shape: _weight(case, seed, at + name + ".weight", *shape)  # noqa: E731
        first_norm, second_norm = w("input_layernorm", hidden), w("post_attention_layernorm", hidden)
        wq, wk, wv = (w("self_attn.%s_proj" % n, c * dim, hidden) for n, c in (("q", heads), ("k", kv_heads), ("v", kv_heads)))
        wo = w("self_attn.o_proj", hidden, heads * dim)
        gate, up, down = w("mlp.gate_proj", ff, hidden), w("mlp.up_proj", ff, hidden), w("mlp.down_proj", hidden, ff)
        for b, x in enumerate(sequences):
            n = x.shape[0]
            keep = 0 if i + 1 < case["layers"] else n - 1  # of the last layer only the last row is asked for
            h = _rms(x, first_norm)
            q, k, v = (h @ wq.T).view(n, heads, dim), (h @ wk.T).view(n, kv_heads, dim), (h @ wv.T).view(n, kv_heads, dim)
            mixed = _attend(turn(q)[keep:], turn(k), v, dim ** -0.5, 0, keep)
            x = x[keep:] + mixed.reshape(n - keep, -1) @ wo.T
            h = _rms(x, second_norm)
            sequences[b] = x + (torch.nn.functional.silu(h @ gate.T) * (h @ up.T)) @ down.T
    last = _rms(torch.stack([x[-1] for x in sequences]), _weight(case, seed, "model.norm.weight", hidden))
    head = embedding if tied else _weight(case, seed, "lm_head.weight", case["vocab"], hidden)
    return last @ head.T


def _exact_moe(case, seed):
    x, tensors = _moe_inputs(case, seed)
    x = x.double()
    w = {name: t.double() for name, t in tensors.items()}
    best = torch.topk(x @ w["router.weight"].T, case["top"], dim=-1)
    share = torch.softmax(best.values, -1)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        weight = (share * (best.indices == e)).sum(-1, keepdim=True)
        at = "experts.%d." % e
        g = (x @ w[at + "gate_proj.weight"].T).clamp(max=7.0)
        u = (x @ w[at + "up_proj.weight"].T).clamp(-7.0, 7.0)
        out += weight * ((g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[at + "down_proj.weight"].T)
    return out


def _exact_scan(case, seed):
    q, k, v, more = _scan_inputs(case, seed)
    repeat = case["heads"] // case["key_heads"]
    q, k = (t.double().repeat_interleave(repeat, 1) for t in (q, k))
    v, more = v.double(), {name: t.double() for name, t in more.items()}
    lengths = _numbers(case["lengths"])
    starts = torch.tensor(np.cumsum([0] + lengths)[:-1].copy(), device="cuda")
    state = torch.zeros(len(lengths), case["heads"], case["dim"], case["vdim"], dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    for t in range(max(lengths)):  # a token of every sequence that still has one
        live = [b for b, n in enumerate(lengths) if t < n]
        at = starts[live] + t
        S, kt, u = state[live], k[at], v[at]
        if "g" in more:
            S = S * more["g"][at][..., None]
            u = more["beta"][at][..., None] * (u - torch.einsum("bhdv,bhd->bhv", S, kt))
        elif "token_decay" in more:
            S = S * more["token_decay"][at][..., None, None]
        else:
            S = S * more["head_decay"][None, :, None, None]
        S = S + kt[..., None] * u[..., None, :]
        out[at] = torch.einsum("bhdv,bhd->bhv", S, q[at])
        state[live] = S
    return out, state


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prompt", "extend"):
        return _exact_model(case, seed)
    if kind == "moe":
        return _exact_moe(case, seed)
    if kind == "scan":
        return _exact_scan(case, seed)
    q, k, v = (t.double() for t in _attention_inputs(case, seed))
    out, at = [], 0
    for n in _numbers(case["lengths"]):
        out.append(_attend(q[at:at + n], k[at:at + n], v[at:at + n], case["dim"] ** -0.5, case["window"], 0))
        at += n
    return torch.cat(out).flatten(1)
