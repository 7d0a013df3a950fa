"""Barriers of the tensor-core kernels, as their sources have them (no GPU needed).

Commits of kernels whose issuing warp stays together around an elected lane: each stands in the lane's block of the products it stands
for. One in an `if` of its own was lost, or came twice, in one of 20 launches of one product. And waits of one lane for its warp."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama_rs_metal_b200", "csrc")


def elected_kernels():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as handle:
                source = re.sub(r"//[^\n]*", "", handle.read())
            if re.search(r"\bumma_commit(_pair)?\(", source) and "elect_one()" in source:
                found.append((name, source))
    return found


KERNELS = elected_kernels()


def block_around(source, at):
    """The innermost braces around a place: the text ahead of them from the last statement on, and what they hold."""
    depth, begin = 0, at
    while True:
        begin -= 1
        depth += {"}": 1, "{": -1}.get(source[begin], 0)
        if depth < 0:
            break
    depth, end = 0, begin
    while True:
        depth += {"{": 1, "}": -1}.get(source[end], 0)
        if depth == 0:
            break
        end += 1
    return source[max(source.rfind(c, 0, begin) for c in ";{}") + 1:begin].strip(), source[begin:end]


def commits(source):
    return [m.start() for m in re.finditer(r"\bumma_commit(_pair)?\(", source)]


def test_the_kernels_are_found():
    assert {"attention_prefill_pingpong.cu", "gemm_bf16_few.cu", "gemm_bf16_umma.cu", "gemm_bf16_umma_pair.cu", "gemm_bf16_wide.cu",
            "gemm_f32_umma.cu"} <= {name for name, _ in KERNELS}


@pytest.mark.parametrize("name,source", KERNELS, ids=[name for name, _ in KERNELS])
def test_commits_stand_with_their_products(name, source):
    names = set(re.findall(r"const bool (\w+) = elect_one\(\);", source))
    lane_of_its_own = 0  # an issuer that is one lane from its start on: its loop over the blocks, and what is behind it
    for at in commits(source):
        head, body = block_around(source, at)
        if head in {"if (%s)" % one for one in names}:
            assert re.search(r"\bumma_bf16\w*\(", body), f"{name}: a commit apart from its products"
        else:
            assert name == "gemm_bf16_umma.cu" and not head.startswith(("if", "else")), f"{name}: a commit under {head!r}"
            lane_of_its_own += 1
    assert lane_of_its_own == (2 if name == "gemm_bf16_umma.cu" else 0)


@pytest.mark.parametrize("name,source", KERNELS, ids=[name for name, _ in KERNELS])
def test_the_arrival_that_is_waited_for_is_the_last(name, source):
    """Nobody waits for the last arrival at a stage, and a CTA leaves when its results have: theirs has to be behind it."""
    both = 0
    for at in commits(source):
        _, body = block_around(source, at)
        told = re.findall(r"\bumma_commit(?:_pair)?\((\w+)", body)
        stages = [i for i, bar in enumerate(told) if bar in ("empty", "kv_free")]
        results = [i for i, bar in enumerate(told) if bar in ("acc_full", "o_done")]
        if stages and results and name != "gemm_f32_umma.cu":  # (there the stage's commit stands for later products, and is waited for)
            both += 1
            assert max(stages) < min(results), f"{name}: {told}"
    assert both or name == "gemm_f32_umma.cu"


@pytest.mark.parametrize("name", ["gemm_bf16_umma_pair.cu", "gemm_bf16_wide.cu"])
def test_no_cta_of_a_pair_leaves_before_its_stages_were_signalled(name):
    """What the leader's commits signal in the other CTA's memory has come before the pair meets for the last time."""
    source = dict(KERNELS)[name]
    last = re.search(r"for \(uint32_t i = it > STAGES \? it - STAGES : 0; i < it && !\*bail; \+\+i\)\s*if \(([^;]*)\) \*bail = 1;", source)
    assert last and "mbar_wait(empty + i % STAGES, (i / STAGES) & 1" in last.group(1)


@pytest.mark.parametrize("function", ["mbar_wait_warp", "ring_ready"])
def test_a_lane_that_waits_for_its_warp_orders_the_others_reads(function):
    """One lane has seen the barrier; a vote tells the others, but only __syncwarp() puts their reads behind what it saw."""
    with open(os.path.join(CSRC, "umma.cuh")) as handle:
        source = handle.read()
    begin = source.index(" %s(" % function)
    body = source[begin:source.index("\n}\n", begin)]
    for vote in re.finditer(r"__(all|ballot|any)_sync\(", body):
        assert "__syncwarp();" in body[vote.end():] and "return __all_sync" not in body
