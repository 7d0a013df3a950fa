"""Row-wise attention in blocks of 32 keys (csrc/attention_rowwise.cu, heads of up to 128) against float64, at the edges of its blocks,
its rows per CTA and its padded head sizes; packed and paged keys give the same bits."""
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randn(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def _int32(x):
    return torch.tensor(list(x), dtype=torch.int32, device=DEV)


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


def _paged(k, v, lengths, page, seed):
    """The sequences' keys and values on pages in disorder, with NaNs where no key is."""
    per = max(-(-n // page) for n in lengths) + 1
    table = torch.randperm(len(lengths) * per, generator=torch.Generator().manual_seed(seed)).int().view(len(lengths), per)
    pages = [torch.full((table.numel(), t.shape[1], page, t.shape[2]), float("nan"), dtype=t.dtype, device=DEV) for t in (k, v)]
    seq, p = (torch.tensor(x) for x in ([b for b, n in enumerate(lengths) for _ in range(n)], [i for n in lengths for i in range(n)]))
    for to, t in zip(pages, (k, v)):
        to[table[seq, p // page].long().to(DEV), :, (p % page).to(DEV)] = t
    return SimpleNamespace(k=pages[0], v=pages[1], page_table=table.to(DEV), kv_heads=k.shape[1], page_size=page, head_dim=k.shape[2],
                           value_dim=None, window=None)


# several sequences in a CTA and one; portions on both sides of 128 queries, to sequences that bring many, few and one each; pages that
# end inside a block of 32 keys; windows that begin inside one; rows off 16 and 8 bytes
@pytest.mark.parametrize("lengths,brought", [([150, 67, 33], [100, 1, 26]), ([150, 67, 33], [100, 1, 27]), ([9] * 65, [2] * 65), ([37, 5] * 70, [1] * 140),
                                             ([40, 64, 1, 70], [1] * 4), ([3] * 129, [1] * 129)])
@pytest.mark.parametrize("heads,kv_heads,d,dv,dtype", [(2, 2, 64, 64, torch.float32), (6, 2, 33, 17, torch.float32), (5, 1, 128, 100, torch.float32),
                                                       (6, 2, 30, 30, torch.bfloat16), (3, 3, 50, 50, torch.bfloat16)])
@pytest.mark.parametrize("window,page,sinks", [(0, 7, False), (40, 48, True), (-48, 20, False)])
def test_paged_rows_have_the_packed_rows_bits(lengths, brought, heads, kv_heads, d, dv, dtype, window, page, sinks):
    from llama_rs_metal_b200.kernels import attention_dispatch, ops
    T = sum(lengths)
    q, k, v = (_randn(T, h, n, seed=h + n).to(dtype) for h, n in ((heads, d), (kv_heads, d), (kv_heads, dv)))
    cu = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    slopes = _randn(heads, seed=9).abs() if sinks else None
    extras = attention_dispatch.Extras(sinks=_randn(heads, seed=8)) if sinks else None
    more = dict(slopes=slopes, extras=extras)
    want = ops.attention_prefill(q, k, v, _int32(cu), _int32([b for b, n in enumerate(lengths) for _ in range(n)]), max(lengths), d ** -0.5, window, **more)
    kv, slots, lens = _paged(k, v, lengths, page, T), _int32(range(len(lengths))), _int32(lengths)
    rows = [cu[b + 1] - n + i for b, n in enumerate(brought) for i in range(n)]
    got = ops.attention_extend(q[rows].contiguous(), kv, _int32([sum(brought[:i]) for i in range(len(brought) + 1)]),
                               _int32([b for b, n in enumerate(brought) for _ in range(n)]),
                               _int32([lengths[b] - n + i for b, n in enumerate(brought) for i in range(n)]), slots, lens, max(brought), d ** -0.5, window, **more)
    assert torch.equal(got, want[rows])
    if set(brought) == {1}:
        assert torch.equal(ops.attention_decode(q[rows].contiguous(), kv, slots, lens, max(lengths), d ** -0.5, window, **more), want[rows])
