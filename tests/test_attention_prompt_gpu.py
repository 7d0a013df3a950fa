"""Attention of prompts on tcgen05 (csrc/attention_prefill_pingpong.cu) in each of its forms, against float64."""
import math

import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# one key; edges of key tiles (64, 128) and query tiles (128, 256); a chain without a tile; packed prompts of unequal length, whose
# tiles are listed (the last three); windows that begin inside and on a key tile
@pytest.mark.parametrize("lengths", [[1], [64], [65], [128, 127], [257], [640, 1], [1300, 1, 64], [1, 1, 900, 129, 256], [1] * 31 + [777]])
@pytest.mark.parametrize("heads,kv_heads,d", [(4, 2, 64), (3, 1, 128)])
@pytest.mark.parametrize("form", [None, "chain", "single", "pingpong"])
@pytest.mark.parametrize("window", [0, 64, 100])
def test_prompts_match_float64(monkeypatch, lengths, heads, kv_heads, d, form, window):
    from llama_rs_metal_b200.kernels import attention_dispatch, gemm_dispatch
    monkeypatch.setattr(attention_dispatch, "prefill_kernel", form)
    gen = torch.Generator().manual_seed(sum(lengths) + d)
    tokens = sum(lengths)
    q = (1.5 * torch.randn(tokens, heads, d, generator=gen)).bfloat16()
    k, v = (torch.randn(tokens, kv_heads, d, generator=gen).bfloat16() for _ in range(2))
    bounds = [sum(lengths[:b]) for b in range(len(lengths) + 1)]
    out = torch.full((tokens, heads, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    owner = torch.tensor([b for b, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32, device=DEV)
    attention_dispatch.prefill(q.to(DEV), k.to(DEV), v.to(DEV), out, torch.tensor(bounds, dtype=torch.int32, device=DEV), owner,
                               max(lengths), 1 / math.sqrt(d), window)
    gemm_dispatch.check_status()
    got = out.double().cpu()
    for begin, end in zip(bounds, bounds[1:]):
        place = torch.arange(end - begin)
        seen = place[None] <= place[:, None]
        if window:
            seen &= place[None] > place[:, None] - window
        for h in range(heads):
            scores = q[begin:end, h].double() @ k[begin:end, h * kv_heads // heads].double().T / math.sqrt(d)
            want = torch.softmax(scores.masked_fill(~seen, -math.inf), -1) @ v[begin:end, h * kv_heads // heads].double()
            # probabilities and results rounded to bfloat16 (2^-9 each), values of size up to four
            assert float((got[begin:end, h] - want).abs().max()) <= 2e-2
