"""State scans of long sequences in blocks of 16 tokens on the tensor cores (csrc/recurrent_block.cuh), at the edges of its blocks, its
tiles of 16 columns, its rows per warp, and of the line to the blocks with FMAs (csrc/recurrent_walk.cuh)."""
import pytest
import torch

from test_state_walk_gpu import DEV, _inputs, _int32, _reference, _run

pytestmark = pytest.mark.gpu

RULES = ["delta", "head_delta", "token_decay", "head_decay", "bonus"]


def _distance(a, b):
    return float((a.double() - b).norm() / b.norm())


# 16 to 1 rows of the last piece of a warp, columns of a whole tile, one more, one; blocks of 16, 15 and one token at the end
@pytest.mark.parametrize("lengths", [[96, 111], [112, 113, 0, 7]])
@pytest.mark.parametrize("H,G,d,dv", [(2, 2, 64, 16), (4, 2, 49, 17), (2, 1, 128, 1), (2, 2, 113, 33), (2, 1, 256, 16), (1, 1, 193, 31),
                                      (6, 1, 16, 8)])
@pytest.mark.parametrize("rule", RULES)
def test_edges_match_the_recurrence_no_further_off_than_token_by_token(rule, H, G, d, dv, lengths):
    G = H if rule == "bonus" else G
    x = _inputs(H, G, d, dv, lengths, seed=d + dv)
    slots = list(range(len(lengths)))
    want, single = _reference(rule, x, lengths, slots), _run(rule, x, lengths, slots, blocks=False)
    for a, b, c in zip(_run(rule, x, lengths, slots), want, single):
        assert _distance(a, b) <= 2e-6                             # float32 sums, forgotten at the decays' rate
        assert _distance(a, b) <= 1.5 * _distance(c, b) + 2.0 ** -26  # both are sums of roundings of 2^-24, those of 16 tokens cut off


# CTAs (tiles x heads x sequences) on both sides of the line: 370 for delta rules, 444 with a bonus or heads of up to 64, 888 with one decay and
# heads of up to 128, 222 for heads beyond
@pytest.mark.parametrize("H,d,dv,seqs", [(46, 64, 64, 2), (47, 64, 64, 2), (55, 64, 64, 2), (56, 64, 64, 2), (37, 160, 48, 2), (38, 160, 48, 2),
                                         (148, 100, 48, 2), (149, 100, 48, 2)])
@pytest.mark.parametrize("rule", RULES)
def test_both_sides_of_the_line_to_the_blocks_with_fmas(rule, H, d, dv, seqs):
    lengths = [97 + 16 * i for i in range(seqs)]
    x = _inputs(H, H, d, dv, lengths, seed=H)
    for a, b in zip(_run(rule, x, lengths, [1, 0]), _reference(rule, x, lengths, [1, 0])):
        assert _distance(a, b) <= 2e-6


@pytest.mark.parametrize("rule", RULES)
def test_inputs_off_16_bytes(rule):
    x = _inputs(3, 3, 64, 24, [130], seed=2)
    moved = {}
    for name, t in x.items():
        room = torch.empty(t.numel() + 1, device=DEV)
        moved[name] = room[1:].view(t.shape).copy_(t)
    for a, b in zip(_run(rule, moved, [130], [0]), _run(rule, x, [130], [0])):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name,value", [("q", float("inf")), ("k", float("nan")), ("v", float("-inf")), ("g", float("nan"))])
@pytest.mark.parametrize("rule", RULES)
def test_what_is_not_finite_shows_where_it_does_token_by_token(rule, name, value):
    """In the second block of eight, in one head and sequence: what comes ahead of it, other heads and the other sequence stay as
    they are, and no read-out that is finite token by token is not."""
    lengths, token = [130, 100], 27
    x = _inputs(2, 2, 64, 20, lengths, seed=7)
    clean, _ = _run(rule, x, lengths, [1, 0])
    x[name][token, 1, 3] = value
    if name == "g":
        x["decay"][token, 1] = value
    got, state = _run(rule, x, lengths, [1, 0])
    want, want_state = _run(rule, x, lengths, [1, 0], blocks=False)
    for a, b in ((got, want), (state, want_state)):
        whole = b.isfinite()
        assert bool(a[whole].isfinite().all()) and _distance(a[whole], b[whole].double()) <= 2e-6
        assert not bool(a[~whole].isfinite().any())
    assert torch.equal(got[:16], clean[:16]) and torch.equal(got[130:], clean[130:])
    assert _distance(got[16:token], clean[16:token].double()) <= 2e-6


# one long sequence among short ones: on the tensor cores where its CTAs alone fit, whatever the step could hold
@pytest.mark.parametrize("lengths", [[300] + [1] * 31, [1, 5, 200, 3], [130, 7, 120, 1, 1]])
@pytest.mark.parametrize("H,d,dv", [(16, 128, 128), (32, 64, 64), (6, 160, 40)])
@pytest.mark.parametrize("rule", RULES)
def test_a_long_sequence_among_short_ones(rule, H, d, dv, lengths):
    x = _inputs(H, H, d, dv, lengths, seed=H + len(lengths))
    slots = [len(lengths) - i for i in range(len(lengths))]
    want = _reference(rule, x, lengths, slots)
    for longest in (max(lengths), 320, None):
        for a, b in zip(_run(rule, x, lengths, slots, longest=longest), want):
            assert _distance(a, b) <= 2e-6


def _still(x, lengths, decay=1.0):
    """Inputs under which nothing is written and the state decays by `decay` alone."""
    for name in ("g", "decay", "head"):
        x[name].fill_(decay)
    x["step"].zero_()
    x["v"].zero_()
    return x


@pytest.mark.parametrize("H,d,dv", [(2, 64, 20), (1, 128, 33), (1, 256, 16)])
@pytest.mark.parametrize("rule", RULES)
def test_a_read_of_one_number_is_rounded_once(rule, H, d, dv):
    """Queries with one number each against a state that stays: single products of float32 numbers."""
    x, T = _still(_inputs(H, H, d, dv, [112], seed=d), [112]), 112
    x["q"] = torch.randn(T, H, d, device=DEV) * (torch.arange(d, device=DEV) == torch.arange(T, device=DEV)[:, None] * 5 % d)[:, None]
    (out, state), (want, _) = _run(rule, x, [112], [1]), _reference(rule, x, [112], [1])
    # the product's rounding; the low parts' product, 2^-34 of it, and the small ones' truncated sum, 2^-31, are left out
    assert bool(((out.double() - want).abs() <= (2.0 ** -24 + 2.0 ** -30) * want.abs()).all())
    assert torch.equal(state, x["state"])


@pytest.mark.parametrize("scale", [2.0 ** -116, 2.0 ** 70])
@pytest.mark.parametrize("H,d,dv", [(2, 64, 20), (1, 128, 33)])
@pytest.mark.parametrize("rule", RULES)
def test_very_small_and_very_large_states(rule, H, d, dv, scale):
    """What is written and held, times a power of two: the same relative distance as token by token."""
    x = _inputs(H, H, d, dv, [120], seed=d + 1)
    x["v"] *= scale
    x["state"] *= scale
    want, single = _reference(rule, x, [120], [1]), _run(rule, x, [120], [1], blocks=False)
    for a, b, c in zip(_run(rule, x, [120], [1]), want, single):
        assert _distance(a / scale, b / scale) <= 1.25 * _distance(c / scale, b / scale) + 2.0 ** -24


@pytest.mark.parametrize("rule", RULES)
def test_keys_and_queries_out_of_the_parts_range(rule):
    """A key and a query of 2^30 and more are read and written with FMAs, the tokens around them as ever."""
    x = _inputs(2, 2, 64, 20, [130], seed=3)
    x["q"][40, 1, 3], x["q"][77, 0, 9] = 2.0 ** 30, 2.0 ** 120
    if rule not in ("delta", "head_delta"):  # (a delta rule's state would grow by the key's square)
        x["k"][55, 0, 5] = 2.0 ** 31
    got, single = _run(rule, x, [130], [1]), _run(rule, x, [130], [1], blocks=False)
    want = _reference(rule, x, [130], [1])
    for a, b, c in zip(got, want, single):
        whole = c.isfinite() & (b.abs() < 2.0 ** 60)
        assert torch.equal(a.isfinite(), c.isfinite())
        assert float((a[whole].double() - b[whole]).norm() / b[whole].norm()) <= 2e-6
