"""Experts of steps of few rows, every chosen expert read once (csrc/moe_rows.cu), against float64."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# rows around the tiles of 8, 16 and 32 pairs, one and more passes over an expert; widths off the tiles of 8 and 16 rows
# and off a warp's share of K; pairs on both sides of 32; the most pairs taken
@pytest.mark.parametrize("T,width,ff,E,top,act,identity", [
    (1, 256, 256, 8, 2, 0, 0), (8, 264, 264, 8, 2, 1, 0), (9, 520, 136, 5, 3, 0, 1), (16, 256, 256, 16, 2, 0, 2),
    (17, 1000, 72, 4, 2, 1, 0), (63, 256, 264, 3, 2, 0, 1), (130, 256, 256, 2, 1, 0, 0), (40, 256, 256, 200, 8, 0, 3),
    (2048, 256, 256, 32, 2, 1, 0), (2049, 256, 256, 32, 2, 1, 0)])
def test_few_rows_match_the_definition_in_float64(T, width, ff, E, top, act, identity):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(T + width)
    limit, alpha = 0.8, 1.702
    gate_up = (torch.randn(E, 2 * ff, width, generator=gen) / width ** 0.5 * 2).bfloat16()
    down = (torch.randn(width, E, ff, generator=gen) / ff ** 0.5).bfloat16()
    x = torch.randn(T, width, generator=gen).bfloat16()
    x32 = torch.randn(T, width, generator=gen)
    ids = torch.stack([torch.randperm(E + identity, generator=gen)[:top] for _ in range(T)]).int()
    weights = torch.rand(T, top, generator=gen)
    planes = ops.moe_experts_rows(x.to(DEV), gate_up.to(DEV), down.to(DEV), ids.to(DEV), weights.to(DEV), limit, alpha, act,
                                  x32.to(DEV) if identity else None)
    if T * top <= 4096:
        assert planes.shape[0] == top  # one plane per choice: the kernel under test ran
    want = torch.zeros(T, width, dtype=torch.float64)
    for e in range(E):
        share = (weights.double() * (ids == e)).sum(1)
        rows = torch.nonzero((ids == e).any(1))[:, 0]
        if rows.numel() == 0:
            continue
        both = x[rows].double() @ gate_up[e].double().T
        g, u = both[:, :ff], both[:, ff:]
        if act == ops.ACT_SILU:
            y = torch.nn.functional.silu(g) * u
        else:
            g = g.clamp(max=limit)
            y = g * torch.sigmoid(alpha * g) * (u.clamp(-limit, limit) + 1)
        want[rows] += share[rows, None] * (y @ down[:, e].double().T)
    want += ((weights.double() * (ids >= E)).sum(1))[:, None] * x32.double()
    got = planes.sum(0, dtype=torch.float64).cpu()
    # float32 throughout: sums of at most 1,000 products, each within a few roundings of 2^-24
    assert float((got - want).norm() / want.norm()) <= 1e-6
    again = ops.moe_experts_rows(x.to(DEV), gate_up.to(DEV), down.to(DEV), ids.to(DEV), weights.to(DEV), limit, alpha, act,
                                 x32.to(DEV) if identity else None)
    assert torch.equal(planes, again)


@pytest.mark.parametrize("T,E", [(591, 8), (592, 8), (594, 9), (5, 32), (5, 16), (700, 40)])
def test_router_gives_a_token_the_same_choice_whatever_shares_its_launch(T, E):
    """Four tokens per CTA and one, and CTAs of 128 to 1,024 threads, add a logit's products in the same order."""
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(T + E)
    x, w = torch.randn(T, 1032, generator=gen).bfloat16().to(DEV), torch.randn(E, 1032, generator=gen).to(DEV)
    ids, weights = ops.moe_router(x, w, None, 3)
    for t in (0, T // 2, T - 1):
        one_ids, one_weights = ops.moe_router(x[t:t + 1].contiguous(), w, None, 3)
        assert torch.equal(one_ids[0], ids[t]) and torch.equal(one_weights[0], weights[t])
    best = torch.topk(x.double() @ w.double().T, 3, dim=-1)
    assert float((torch.softmax(best.values, -1) - weights).abs().max()) <= 2e-4  # logits of some 30, each within 1e-4
