"""State scans of long sequences, eight or four tokens at a time (csrc/recurrent_walk.cuh), against float64 token by token."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


def _int32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


# head sizes on both sides of 64, 128 and 256, value widths off a CTA's columns and off 16 bytes, few and many heads
# (four and eight rows per thread, two and four columns, of each padded size); lengths on both sides of a block of 4 or 8 and a stage of 16, none, and
# one token among long ones
SHAPES = [(2, 1, 64, 32), (3, 3, 33, 17), (12, 4, 65, 50), (4, 2, 128, 128), (16, 4, 128, 144), (2, 2, 129, 9), (1, 1, 256, 24),
          (24, 24, 64, 64), (40, 8, 128, 96), (48, 48, 64, 64), (64, 8, 33, 50)]
LENGTHS = [[96], [97, 191, 1], [200, 0, 107], [95, 111]]


def _inputs(H, G, d, dv, lengths, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *shape: torch.rand(*shape, generator=gen, device=DEV)  # noqa: E731
    randn = lambda *shape: torch.randn(*shape, generator=gen, device=DEV)  # noqa: E731
    T = sum(lengths)
    unit = torch.nn.functional.normalize
    q, k = unit(randn(T, G, d), dim=-1), unit(randn(T, G, d), dim=-1)
    g = 1 - 0.5 * rand(T, H, d)
    g[:, 0, : d // 2] = 1e-4 * rand(T, d // 2)  # decays whose product over a block underflows towards nothing
    return dict(q=q, k=k, v=randn(T, H, dv), g=g, decay=1 - 0.5 * rand(T, H), step=rand(T, H), head=1 - 0.5 * rand(H),
                bonus=randn(H, d), state=randn(len(lengths) + 1, H, d, dv))


def _reference(rule, x, lengths, slots):
    x = {name: t.double() for name, t in x.items()}
    H, G = x["v"].shape[1], x["q"].shape[1]
    out, state, at = torch.empty_like(x["v"]), x["state"].clone(), 0
    for n, slot in zip(lengths, slots):
        S = state[slot].clone() if slot >= 0 else torch.zeros_like(state[0])
        for t in range(at, at + n):
            q, k, v = x["q"][t].repeat_interleave(H // G, 0), x["k"][t].repeat_interleave(H // G, 0), x["v"][t]
            if rule == "bonus":
                out[t] = torch.einsum("hdv,hd->hv", S + (x["bonus"] * k)[..., None] * v[:, None], q)
                S = S * x["g"][t][..., None] + k[..., None] * v[:, None]
                continue
            decay = {"delta": x["g"][t][..., None], "token_decay": x["decay"][t][:, None, None],
                     "head_delta": x["decay"][t][:, None, None], "head_decay": x["head"][:, None, None]}[rule]
            S = S * decay
            if rule in ("delta", "head_delta"):
                v = x["step"][t][:, None] * (v - torch.einsum("hdv,hd->hv", S, k))
            S = S + k[..., None] * v[:, None]
            out[t] = torch.einsum("hdv,hd->hv", S, q)
        if slot >= 0:
            state[slot] = S
        at += n
    return out, state


def _run(rule, x, lengths, slots, **options):
    from llama_rs_metal_b200.kernels import ops
    state, cu = x["state"].clone(), _int32([sum(lengths[:i]) for i in range(len(lengths) + 1)])
    H, d, dv = x["bonus"].shape[0], x["bonus"].shape[1], x["v"].shape[2]
    if rule == "bonus":  # q, k and v as columns of a wider activation
        T = x["q"].shape[0]
        proj = torch.cat([x["q"].reshape(T, -1), torch.zeros(T, 3, device=DEV), x["k"].reshape(T, -1), x["v"].reshape(T, -1)], dim=1)
        out = ops.bonus_state_scan(proj.contiguous(), 0, H * d + 3, 2 * H * d + 3, x["g"].reshape(T, -1).contiguous(), x["bonus"],
                                   state, cu, _int32(slots), dv, **options)
    elif rule == "head_delta":
        out = ops.head_decay_delta_scan(x["q"], x["k"], x["v"], x["decay"], x["step"], state, cu, _int32(slots), **options)
    else:
        more = {"delta": dict(g=x["g"], beta=x["step"]), "token_decay": dict(token_decay=x["decay"]),
                "head_decay": dict(head_decay=x["head"])}[rule]
        out = ops.linear_state_scan(x["q"], x["k"], x["v"], state, cu, _int32(slots), **more, **options)
    return out, state


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("H,G,d,dv", SHAPES)
@pytest.mark.parametrize("rule", ["delta", "head_delta", "token_decay", "head_decay", "bonus"])
def test_long_walks_match_the_recurrence(rule, H, G, d, dv, lengths):
    if rule == "bonus":
        G = H
    x = _inputs(H, G, d, dv, lengths, seed=d + dv + len(lengths))
    slots = [len(lengths) - i for i in range(len(lengths))]
    got, want = _run(rule, x, lengths, slots), _reference(rule, x, lengths, slots)
    for a, b in zip(got, want):  # float32 sums of up to d terms, forgotten at the decays' rate
        assert float((a.double() - b).norm() / b.norm()) <= 2e-6
    untouched = [s for s in range(len(lengths) + 1) if s not in slots]
    assert all(torch.equal(got[1][s], x["state"][s]) for s in untouched)


@pytest.mark.parametrize("rule", ["delta", "head_delta", "token_decay", "bonus"])
def test_a_token_takes_nothing_from_the_tokens_behind_it(rule):
    """A NaN in token 21 leaves every earlier token's read-out alone, whatever block it shares; a sequence of padding (slot
    -1) starts from nothing and stores nothing."""
    x = _inputs(2, 2, 64, 32, [112, 90], seed=1)
    clean, _ = _run(rule, x, [112, 90], [0, -1])
    want, _ = _reference(rule, x, [112, 90], [0, -1])
    assert float((clean.double() - want).norm() / want.norm()) <= 2e-6
    x["v"][21] = float("nan")
    spoilt, state = _run(rule, x, [112, 90], [0, -1])
    assert torch.equal(spoilt[:21], clean[:21]) and torch.equal(spoilt[112:], clean[112:])
    assert bool(spoilt[22:112].isnan().all()) and bool(state[0].isnan().all())
    assert torch.equal(state[1:], x["state"][1:])


@pytest.mark.parametrize("rule", ["token_decay", "head_decay", "bonus"])
@pytest.mark.parametrize("H,d,dv", [(2, 64, 32), (16, 128, 144), (40, 128, 96)])
def test_an_infinite_state_stays_infinite_and_alone(rule, H, d, dv):
    """Without a delta rule an infinity in the state stays where it is, under decays of one and below, and shows in the
    read-outs of its column only."""
    lengths, slots = [101, 112], [1, 2]
    x = _inputs(H, H, d, dv, lengths, seed=5)
    x["g"].clamp_(min=0.5)  # no block's decays underflow: infinity times nothing would not be a number
    for name in ("g", "decay"):
        x[name][::3] = 1.0
    x["head"][0] = 1.0
    x["state"][1, 0, 3, 5], x["state"][2, H - 1, d - 1, dv - 1] = float("inf"), float("-inf")
    got, want = _run(rule, x, lengths, slots), _reference(rule, x, lengths, slots)
    for a, b in zip(got, want):
        whole = b.isfinite()
        assert bool((~whole).any()) and torch.equal(a[~whole].double(), b[~whole])
        assert float((a[whole].double() - b[whole]).norm() / b[whole].norm()) <= 2e-6


def _cut(x, begin, end):
    return {name: t if name in ("head", "bonus", "state") else t[begin:end].contiguous() for name, t in x.items()}


@pytest.mark.parametrize("rule", ["delta", "head_delta", "token_decay", "head_decay", "bonus"])
def test_without_blocks_cuts_and_company_change_no_bit(rule):
    """Whole, in portions on both sides of the line to the blocked form, and beside other sequences."""
    x = _inputs(40, 40, 64, 80, [300, 40, 129], seed=3)
    (out, state), (alone, alone_state) = (_run(rule, y, n, s, blocks=False) for y, n, s in
                                          ((x, [300, 40, 129], [1, 2, 3]), (_cut(x, 0, 300), [300], [1])))
    assert torch.equal(out[:300], alone) and torch.equal(state[1], alone_state[1])
    held, parts = x, []
    for begin, end in ((0, 97), (97, 98), (98, 300)):
        o, s = _run(rule, dict(_cut(held, begin, end)), [end - begin], [1], blocks=False)
        held = dict(held, state=s)
        parts.append(o)
    assert torch.equal(torch.cat(parts), alone) and torch.equal(held["state"][1], alone_state[1])


@pytest.mark.parametrize("rule", ["delta", "head_delta", "token_decay", "head_decay", "bonus"])
@pytest.mark.parametrize("lengths", [[30, 500, 95, 96], [3, 200, 1, 2, 96, 5, 1] + [1] * 30 + [97]])
def test_a_sequence_goes_its_way_whatever_the_others_bring(rule, lengths):
    """Each sequence's own tokens decide between blocks and token by token (96 tokens; heads enough for one layout either
    way), where the tokens let all walk and where the kernel finds those that do; a hint of the longest only saves launches."""
    x = _inputs(80, 80, 64, 96, lengths, seed=4)
    slots = list(range(1, len(lengths) + 1))
    out, state = _run(rule, x, lengths, slots)
    at = 0
    for n, slot in zip(lengths, slots):
        for options in ({}, dict(longest=n)):
            alone, alone_state = _run(rule, _cut(x, at, at + n), [n], [slot], **options)
            assert torch.equal(out[at:at + n], alone) and torch.equal(state[slot], alone_state[slot])
        at += n
    few = _cut(x, at - 191, at)  # no sequence in blocks, with the launches for them and without
    assert all(torch.equal(a, b) for a, b in zip(_run(rule, few, [95, 90, 6], [3, 4, 0]),
                                                 _run(rule, few, [95, 90, 6], [3, 4, 0], longest=95)))


@pytest.mark.parametrize("rule", ["delta", "head_delta", "token_decay", "head_decay", "bonus"])
@pytest.mark.parametrize("H,d,dv", [(4, 64, 32), (3, 128, 40), (2, 200, 24)])
def test_a_bounded_workspace_changes_no_bit(monkeypatch, rule, H, d, dv):
    """In pieces of several sequences and of one, of many stages and of one; with padding, a short sequence and an empty one
    among them. The scratch is no larger than allowed, or than a stage."""
    from llama_rs_metal_b200.kernels import ops
    lengths, slots = [130, 0, 400, 20, 112, 97], [1, 2, 3, 4, -1, 5]
    x = _inputs(H, H, d, dv, lengths, seed=6)
    want, held = _run(rule, x, lengths, slots), []
    made = ops._walk_workspace
    monkeypatch.setattr(ops, "_walk_workspace", lambda *a: held.append(made(*a)) or held[-1])
    _run(rule, x, lengths, slots)
    whole, stages = held[-1].numel(), sum(lengths) // 16 + len(lengths)
    for room in (stages - 1, 20, 7, 1, 0):
        monkeypatch.setattr(ops, "SCAN_FLOATS", room * (whole // stages) + 3)
        out, state = _run(rule, x, lengths, slots)
        assert torch.equal(state, want[1]) and torch.equal(out[:550], want[0][:550]) and torch.equal(out[662:], want[0][662:])
        assert float((out[550:662] - want[0][550:662]).norm() / want[0][550:662].norm()) <= 2e-6  # padding: token by token
        assert held[-1].numel() <= max(1, room) * (whole // stages) + 3
