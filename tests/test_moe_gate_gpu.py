"""The gate of sorted experts in the first product's epilogue (csrc/gemm_bf16_umma.cu GATED), and the router's choice by a warp
(csrc/moe.cu choose_top)."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# ff on and off a tile's 128 gate columns; more tiles than SMs; values on both sides of the quotient's lines, no weight
@pytest.mark.parametrize("T,width,ff,E,top,act", [(70, 64, 64, 3, 2, 0), (300, 128, 128, 4, 1, 1), (513, 64, 192, 5, 2, 1),
                                                  (700, 192, 320, 4, 3, 0), (4096, 64, 1024, 8, 2, 1)])
@pytest.mark.parametrize("scale", [1.0, 40.0])
def test_the_same_bits_as_a_gate_of_its_own(monkeypatch, T, width, ff, E, top, act, scale):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    gen = torch.Generator().manual_seed(T + ff)
    gate_up = (torch.randn(E, 2 * ff, width, generator=gen) * scale / width ** 0.5).bfloat16().to(DEV)
    down = (torch.randn(width, E, ff, generator=gen) / ff ** 0.5).bfloat16().to(DEV)
    x = torch.randn(T, width, generator=gen).bfloat16().to(DEV)
    ids = torch.topk(torch.rand(T, E, generator=gen), top).indices.int().to(DEV)
    weights = torch.rand(T, top, generator=gen).to(DEV)
    weights[::7] = 0.0
    got = ops.moe_experts_sorted(x, gate_up, down, ids, weights, 7.0, 1.702, act)
    monkeypatch.setattr(gemm_dispatch, "no_fused_gate", True)
    want = ops.moe_experts_sorted(x, gate_up, down, ids, weights, 7.0, 1.702, act)
    gemm_dispatch.check_status()
    # g exp(g) below -80 for g / (1 + exp(-g)): under 1e-31 either way, nothing in a sum of ordinary numbers
    assert torch.equal(got, want)


def serial_choice(z, top):
    """The largest of what is left, the first of equals; a NaN that comes first stays (nothing is larger)."""
    ids, left = [], list(range(len(z)))
    for _ in range(top):
        best = left[0]
        for e in left[1:]:
            if z[e] > z[best]:
                best = e
        ids.append(best)
        left.remove(best)
    return ids


# outputs below, at and over a warp's lanes, every one chosen, more than 32 choices; one and four tokens to a CTA; a width off the
# steps of 512 and off pairs
@pytest.mark.parametrize("T,E,top,width", [(3, 1, 1, 64), (5, 8, 2, 520), (700, 8, 8, 2048), (601, 33, 3, 515), (9, 128, 40, 1024),
                                           (600, 32, 32, 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_routers_choice(T, E, top, width, dtype):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(E + width)
    x = torch.randint(-3, 4, (T, width), generator=gen).to(dtype)
    w = torch.randint(-1, 2, (E, width), generator=gen).float()  # whole numbers: exact logits, and ties
    bias = torch.randint(-2, 3, (E,), generator=gen).float()
    if E > 4:
        bias[2], bias[4] = float("-inf"), float("inf")
    special = x.clone()
    if T > 4:
        special[1, 0] = float("nan")  # every logit
    ids, weights = ops.moe_router(special.to(DEV), w.to(DEV), bias.to(DEV), top)
    logits = special.double() @ w.double().T + bias.double()
    for t in range(T):
        want = serial_choice(logits[t].tolist(), top)
        assert ids[t].tolist() == want
        share = torch.exp(logits[t][want] - logits[t][want[0]])
        share = share / share.sum()
        same = (weights[t].double().cpu() - share).abs() <= 1e-6
        assert bool((same | (weights[t].cpu().isnan() & share.isnan())).all())


# the gated values themselves: gates over the whole range and at its ends, in rows with a weight, without one and without a pair
@pytest.mark.parametrize("act,alpha", [(1, 1.0), (0, 1.702)])
def test_the_gated_values_are_the_bits_of_a_gate_of_its_own(act, alpha):
    import ctypes
    from llama_rs_metal_b200.kernels import gemm_dispatch, library
    from llama_rs_metal_b200.kernels.ops import _ptr, _stream
    lib, E, ff, K, tiles = library.load(), 2, 128, 64, 3
    M = tiles * 128
    edges = [0.0, -0.0, 1e-38, -1e-38, 79.5, -79.5, 80.0, -80.0, 80.5, -80.5, -88.0, -88.5, -89.0, -104.0, 1e4, -1e4, 3e38, -3e38]
    gates = torch.cat([torch.tensor(edges), torch.linspace(-110, 12, E * ff - len(edges) - 2), torch.tensor([float("inf"), float("-inf")])])
    gate_up = torch.zeros(E, 2, ff, K)
    gate_up[:, 0, :, 0], gate_up[:, 1, :, 0] = (gates / alpha).view(E, ff), torch.linspace(-2, 2, E * ff).view(E, ff)
    x = torch.zeros(M, K)
    x[:, 0] = torch.linspace(0.5, 1.0, M)
    x, gate_up = x.bfloat16().to(DEV), gate_up.bfloat16().view(E * 2 * ff, K).contiguous().to(DEV)
    rows = torch.arange(M, dtype=torch.int32)
    rows[5::9] = -1
    weights = torch.linspace(-1, 1, M)
    weights[3::7] = 0.0
    rows, weights, experts = rows.to(DEV), weights.to(DEV), torch.tensor([0, 1, 1], dtype=torch.int32, device=DEV)
    status = _ptr(gemm_dispatch._status_word(x.device))
    gemm_dispatch.mark_status_dirty()
    both, want, got = (torch.zeros(M, n, dtype=t, device=DEV) for n, t in ((2 * ff, torch.float32), (ff, torch.bfloat16), (ff, torch.bfloat16)))
    tail = (ctypes.c_float(7.0), ctypes.c_float(alpha), act)
    assert lib.lrm_gemm_bf16_umma_experts(_ptr(x), _ptr(gate_up), _ptr(both), M, 2 * ff, K, ctypes.c_longlong(E * 2 * ff), ctypes.c_longlong(K),
                                          2 * ff, 0, _ptr(experts), status, _stream()) == 0
    assert lib.lrm_moe_sorted_gate(_ptr(both), _ptr(rows), _ptr(experts), _ptr(weights), ff, tiles, *tail, _ptr(want), _stream()) == 0
    assert lib.lrm_gemm_bf16_umma_experts_gated(_ptr(x), _ptr(gate_up), _ptr(got), M, ff, K, ctypes.c_longlong(E * 2 * ff), _ptr(experts),
                                                _ptr(rows), _ptr(weights), *tail, status, _stream()) == 0
    gemm_dispatch.check_status()
    same = (got.view(torch.int16) == want.view(torch.int16)) | (got.isnan() & want.isnan())
    gate = both[:, :ff].clamp(max=7.0 if act == 0 else float("inf"))
    # Below -80 the quotient is g exp(z), which is there yet where the division's denominator is infinite (from -88.8 on): apart by
    # the exponentials' roundings and bfloat16's, and by what the division loses, |g| exp(-88.7) < 1e-36 times the rest.
    rest = (both[:, ff:].abs() + 1) * weights[:, None].abs()
    far = (got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 1e-36 * rest
    assert bool((same | ((alpha * gate < -80) & far)).all()) and bool((alpha * gate < -80).any())
