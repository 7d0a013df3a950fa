"""Attention of portions over the paged cache on tcgen05 (csrc/attention_prefill_pingpong.cu, PAGED), against float64."""
import math

import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# held and new tokens around pages of 64 keys and query tiles of 128; a sequence at its start; one new token; windows that
# begin inside and on a page
@pytest.mark.parametrize("held,new", [([0], [65]), ([1], [127]), ([63], [129]), ([64, 1000], [128, 64]), ([700, 0, 5], [300, 1, 66]),
                                      ([129, 61], [2, 257])])
@pytest.mark.parametrize("heads,kv_heads,d", [(8, 2, 64), (4, 4, 128), (6, 2, 128)])
@pytest.mark.parametrize("window", [None, 64, 100])
def test_portions_match_float64(monkeypatch, held, new, heads, kv_heads, d, window):
    from llama_rs_metal_b200.cache.cache import KeyValueView
    from llama_rs_metal_b200.kernels import attention_dispatch, gemm_dispatch, ops
    monkeypatch.setattr(attention_dispatch, "EXTEND_UMMA_CTAS", 1)
    took, rule = [], attention_dispatch.extends_on_tcgen05
    monkeypatch.setattr(attention_dispatch, "extends_on_tcgen05", lambda *a: took.append(rule(*a)) or took[-1])
    gen = torch.Generator().manual_seed(sum(held) + d)
    lengths = [h + n for h, n in zip(held, new)]
    per = max(-(-n // 64) for n in lengths)
    pages = sum(-(-n // 64) for n in lengths) + 3
    order = torch.randperm(pages, generator=gen).tolist()
    table = torch.full((len(new) + 1, per), -1, dtype=torch.int32)
    slots = list(range(len(new), 0, -1))
    # rows that hold no key are what an earlier owner left there: not a number, here
    k = torch.full((pages, kv_heads, 64, d), float("nan"))
    v = torch.full((pages, kv_heads, 64, d), float("nan"))
    q = torch.randn(sum(new), heads, d, generator=gen).bfloat16()
    want, at = [], 0
    for b, (n, length) in enumerate(zip(new, lengths)):
        keys = torch.randn(length, kv_heads, d, generator=gen).bfloat16()
        values = torch.randn(length, kv_heads, d, generator=gen).bfloat16()
        first = 0 if window is None else max(0, held[b] - window + 1) // 64
        for i in range(first, -(-length // 64)):  # pages wholly before the first query's window are not there
            table[slots[b], i] = order.pop()
            rows = slice(64 * i, min(64 * i + 64, length))
            k[table[slots[b], i], :, : rows.stop - rows.start] = keys[rows].transpose(0, 1).float()
            v[table[slots[b], i], :, : rows.stop - rows.start] = values[rows].transpose(0, 1).float()
        place = torch.arange(held[b], length)[:, None]
        seen = torch.arange(length)[None] <= place
        if window is not None:
            seen &= torch.arange(length)[None] > place - window
        for h in range(heads):
            scores = q[at:at + n, h].double() @ keys[:, h * kv_heads // heads].double().T / math.sqrt(d)
            want.append(torch.softmax(scores.masked_fill(~seen, -math.inf), -1) @ values[:, h * kv_heads // heads].double())
        at += n
    int32 = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)  # noqa: E731
    view = KeyValueView(k.bfloat16().to(DEV), v.bfloat16().to(DEV), table.to(DEV), 64, kv_heads, d, window)
    got = ops.attention_extend(q.to(DEV), view, int32([sum(new[:b]) for b in range(len(new) + 1)]),
                               int32([b for b, n in enumerate(new) for _ in range(n)]),
                               int32([p for h, n in zip(held, new) for p in range(h, h + n)]), int32(slots), int32(lengths),
                               max(new), 1 / math.sqrt(d), window).view(-1, heads, d).double().cpu()
    assert took == [True]
    gemm_dispatch.check_status()
    at, left = 0, iter(want)
    for n in new:
        expected = torch.stack([next(left) for _ in range(heads)], 1)
        # probabilities and results rounded to bfloat16 (2^-9 each), values of size one
        assert float((got[at:at + n] - expected).abs().max()) <= 2e-2
        assert float((got[at:at + n] - expected).norm() / expected.norm()) <= 4e-3
        at += n
