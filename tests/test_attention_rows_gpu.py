"""Row-wise attention in blocks of 32 keys (csrc/attention_rowwise.cu, heads of up to 128) against float64, at the edges of its blocks,
its rows per CTA and its padded head sizes; packed and paged keys give the same bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randn(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def _int32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _reference(q, k, v, lengths, scale, window):
    out, at, group = [], 0, q.shape[1] // k.shape[1]
    for n in lengths:
        p = torch.arange(n, device=DEV)
        first = (p - window + 1).clamp(min=0) if window > 0 else (p - p % -window if window < 0 else p * 0)
        hidden = (p[None, :] > p[:, None]) | (p[None, :] < first[:, None])
        kk, vv = (t[at:at + n].double().repeat_interleave(group, 1) for t in (k, v))
        scores = (torch.einsum("qhd,khd->hqk", q[at:at + n].double(), kk) * scale).masked_fill(hidden, -math.inf)
        out.append(torch.einsum("hqk,khd->qhd", torch.softmax(scores, -1), vv))
        at += n
    return torch.cat(out).flatten(1)


# sequences that end at, before and behind a block of 32 keys; rows of several sequences in a CTA; heads that share keys alone, by three, by five
@pytest.mark.parametrize("lengths", [[1], [31, 33, 1, 64], [97, 160]])
@pytest.mark.parametrize("heads,kv_heads,d,dv", [(4, 4, 64, 64), (6, 2, 64, 64), (10, 2, 33, 17), (3, 1, 128, 128), (2, 2, 65, 100), (2, 1, 5, 3)])
@pytest.mark.parametrize("window", [0, 40, -48])
def test_packed_rows_match_float64(lengths, heads, kv_heads, d, dv, window):
    from llama_rs_metal_b200.kernels import ops
    T = sum(lengths)
    q, k, v = _randn(T, heads, d), _randn(T, kv_heads, d, seed=1), _randn(T, kv_heads, dv, seed=2)
    cu = _int32([sum(lengths[:i]) for i in range(len(lengths) + 1)])
    seq = _int32([i for i, n in enumerate(lengths) for _ in range(n)])
    got = ops.attention_prefill(q, k, v, cu, seq, max(lengths), d ** -0.5, window)
    want = _reference(q, k, v, lengths, d ** -0.5, window)
    assert float((got.double() - want).abs().max()) <= 1e-5 * float(v.abs().max())  # roundings of some 200 weighted sums


def test_a_row_takes_nothing_from_keys_it_does_not_see():
    from llama_rs_metal_b200.kernels import ops
    q, k, v = (_randn(70, h, 64, seed=h) for h in (4, 2, 2))
    run = lambda: ops.attention_prefill(q, k, v, _int32([0, 40, 70]), _int32([0] * 40 + [1] * 30), 40, 0.125, None)  # noqa: E731
    clean = run()
    k[20], v[20] = float("nan"), float("inf")
    spoilt = run()
    assert torch.equal(spoilt[:20], clean[:20]) and torch.equal(spoilt[40:], clean[40:])
    assert not bool(spoilt[20:40].isfinite().any())
