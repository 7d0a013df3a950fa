"""Prompt attention on tcgen05 (csrc/attention_prefill_pingpong.cu), launched again and again: every stage and every chain's end reaches
who waits for it, every time."""
import math

import pytest
import torch

DEV = "cuda"


# many short and unequal prompts, whose CTAs end one after another, and rings that go round several times
@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [[1, 65, 700, 64, 129, 900, 3, 257] * 3, [40] * 64, [1500, 31, 1200]])
@pytest.mark.parametrize("heads,kv_heads,d", [(16, 4, 64), (12, 4, 128)])
@pytest.mark.parametrize("form", ["chain", "single", "pingpong"])
def test_every_launch_is_the_first(monkeypatch, lengths, heads, kv_heads, d, form):
    from llama_rs_metal_b200.kernels import attention_dispatch, gemm_dispatch
    monkeypatch.setattr(attention_dispatch, "prefill_kernel", form)
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + d)
    tokens = sum(lengths)
    q, k, v = (torch.randn(tokens, n, d, generator=gen, device=DEV).bfloat16() for n in (heads, kv_heads, kv_heads))
    bounds = [sum(lengths[:b]) for b in range(len(lengths) + 1)]
    cu = torch.tensor(bounds, dtype=torch.int32, device=DEV)
    owner = torch.tensor([b for b, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32, device=DEV)
    want = torch.empty(tokens, heads, d, dtype=torch.float64, device=DEV)
    for begin, end in zip(bounds, bounds[1:]):
        hidden = torch.ones(end - begin, end - begin, dtype=torch.bool, device=DEV).triu(1)
        for h in range(heads):
            scores = q[begin:end, h].double() @ k[begin:end, h * kv_heads // heads].double().T / math.sqrt(d)
            want[begin:end, h] = torch.softmax(scores.masked_fill(hidden, -math.inf), -1) @ v[begin:end, h * kv_heads // heads].double()
    first = None
    for rep in range(100):  # the product that lost one did so in one of 20 launches
        out = torch.full((tokens, heads, d), float("nan"), dtype=torch.bfloat16, device=DEV)
        attention_dispatch.prefill(q, k, v, out, cu, owner, max(lengths), 1 / math.sqrt(d), 0)
        if first is None:
            first = out
            # probabilities and results rounded to bfloat16 (2^-9 each), values of size up to five
            assert float((out.double() - want).abs().max()) <= 2.5e-2
        assert torch.equal(out, first), f"launch {rep}"
    gemm_dispatch.check_status()
