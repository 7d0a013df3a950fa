"""Which way a step's state scans go (csrc/recurrent_block.cuh block_takes_fma): read off the workspace the library asks for."""
import pytest

WALK, STAGE = 96, 16


def _stage_floats(rule, H, d, dv, lengths, longest):
    """Floats of a stage of 16 tokens, which differ between the tensor cores' blocks and those with FMAs."""
    from llama_rs_metal_b200.kernels import library
    lib, tokens = library.load(), sum(lengths)
    if rule == "bonus":
        floats = lib.lrm_bonus_state_scan_floats(len(lengths), H, d, dv, tokens, longest)
    elif rule == "head_delta":
        floats = lib.lrm_head_decay_delta_scan_floats(len(lengths), H, H, d, dv, tokens, longest)
    else:
        floats = lib.lrm_linear_state_scan_floats({"head_decay": 0, "delta": 1, "token_decay": 2}[rule], len(lengths), H, H, d, dv, tokens, longest)
    stages = tokens // STAGE + len(lengths)
    assert floats > 0 and floats % stages == 0
    return floats // stages


# heads whose lone walk fits the SMs; per rule, of each padded size
HEADS = [("delta", 8, 128, 128), ("delta", 16, 128, 128), ("delta", 16, 200, 64), ("head_delta", 16, 128, 128), ("head_delta", 8, 256, 64),
         ("bonus", 32, 64, 64), ("bonus", 16, 128, 128), ("token_decay", 16, 256, 64), ("head_decay", 16, 129, 64),
         ("token_decay", 16, 128, 128), ("head_decay", 32, 64, 64)]


@pytest.mark.parametrize("rule,H,d,dv", HEADS)
@pytest.mark.parametrize("short", [[1] * 31, [1] * 3, [1], [95, 40, 1], [20] * 60])
def test_a_long_sequence_goes_as_it_does_alone_whatever_stands_beside_it(rule, H, d, dv, short):
    lone = _stage_floats(rule, H, d, dv, [2048], 2048)
    assert _stage_floats(rule, H, d, dv, [2048] + short, 2048) == lone
    assert _stage_floats(rule, H, d, dv, [1] + [2048] + short, 2112) == lone  # a bound of the longest, as padded steps know it
    if 2048 + sum(short) < (len(short) + 1) * WALK:  # not known: told by the average
        assert _stage_floats(rule, H, d, dv, [2048] + short, 0) == lone


@pytest.mark.parametrize("rule,H,d,dv", HEADS)
def test_many_long_sequences_go_with_fmas(rule, H, d, dv):
    lone = _stage_floats(rule, H, d, dv, [2048], 2048)
    for longest in (256, 0):
        assert _stage_floats(rule, H, d, dv, [256] * 16, longest) != lone


@pytest.mark.parametrize("rule", ["token_decay", "head_decay"])
def test_one_decay_a_token_goes_with_fmas_where_their_ctas_fill_the_sms(rule):
    way = lambda seqs, longest=600: _stage_floats(rule, 16, 128, 128, [600] * seqs, longest)  # noqa: E731
    lone = way(1)
    assert [way(n) != lone for n in (2, 3, 4, 5, 6, 8)] == [False, False, True, False, False, True]
    assert way(4, 0) == lone


# two prompts of 2,048 tokens beside one another: what the blocks with FMAs held in 64 Mi floats, the tensor cores' larger stages hold too
@pytest.mark.parametrize("rule,H,d,dv", HEADS)
def test_two_prompts_go_whole(rule, H, d, dv):
    from llama_rs_metal_b200.kernels import ops
    lengths = [2048, 2048, 1, 1]
    assert _stage_floats(rule, H, d, dv, lengths, 2048) * (sum(lengths) // STAGE + len(lengths)) <= ops.SCAN_FLOATS
