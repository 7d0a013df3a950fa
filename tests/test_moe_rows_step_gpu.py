"""A mixture's step of few rows in one call (lrm_moe_rows_step): the same bits as router, experts and sum one by one, with the experts
numbered by the choices or, from twice as many pairs as experts on, by themselves."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,width,ff,experts,top,identity,scored", [
    (1, 512, 128, 8, 2, 0, False), (8, 2048, 1024, 8, 2, 0, False), (7, 520, 136, 8, 2, 0, False), (8, 512, 128, 9, 2, 0, False),
    (17, 512, 256, 16, 4, 0, False), (63, 512, 128, 4, 1, 0, False), (40, 264, 264, 32, 3, 0, True), (33, 512, 128, 8, 4, 5, True),
    (3, 512, 128, 5, 2, 3, True), (16, 512, 136, 1, 1, 0, False), (300, 512, 128, 64, 2, 0, False)])
@pytest.mark.parametrize("crowded", [False, True])  # every token chooses the same few experts: the others have no pair
def test_the_same_bits(tokens, width, ff, experts, top, identity, scored, crowded):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(tokens + width)
    x = torch.randn(tokens, width, generator=gen, device=DEV).bfloat16()
    if crowded:
        x = x[:1].repeat(tokens, 1).contiguous()
    router = torch.randn(experts + identity, width, generator=gen, device=DEV) * 0.05
    bias = None if scored else torch.randn(experts, generator=gen, device=DEV)
    gate_up = (torch.randn(experts, 2 * ff, width, generator=gen, device=DEV) * 0.05).bfloat16()
    down = (torch.randn(width, experts, ff, generator=gen, device=DEV) * 0.05).bfloat16()
    scoring = ops.Scoring(torch.randn(experts + identity, generator=gen, device=DEV) * 0.01, 1, 1, True, 1e-6, 2.0) if scored else None
    x32 = torch.randn(tokens, width, generator=gen, device=DEV) if identity else None
    ids, weights = ops.moe_router(x, router, bias, top, scoring)
    want = ops.moe_experts_rows(x, gate_up, down, ids, weights, 7.0, 1.702, 0, x32)
    got = ops.moe_rows_step(x, router, bias, top, scoring, gate_up, down, 7.0, 1.702, 0, x32)
    assert torch.equal(got, want)
    total = want[0].clone()
    if top > 1:
        ops.add_planes_(total, want[1:].contiguous())
    assert torch.equal(ops.moe_rows_step(x, router, bias, top, scoring, gate_up, down, 7.0, 1.702, 0, x32, sum_planes=True), total)
    # against float64: three bfloat16 terms of y and float32 sums of at most width or ff products
    dense = torch.zeros(tokens, width, dtype=torch.float64, device=DEV)
    size = torch.zeros_like(dense)
    for t in range(tokens):
        for c in range(top):
            e, weight = int(ids[t, c]), float(weights[t, c])
            if e >= experts:
                dense[t] += weight * x32[t].double()
                size[t] += weight * x32[t].double().abs()
                continue
            both = gate_up[e].double() @ x[t].double()
            g, u = both[:ff].clamp(max=7.0), both[ff:].clamp(-7.0, 7.0)
            y = g * torch.sigmoid(1.702 * g) * (u + 1)
            dense[t] += weight * (down[:, e].double() @ y)
            size[t] += weight * (down[:, e].double().abs() @ (y.abs() + gate_up[e].double().abs()[:ff] @ x[t].double().abs()))
    assert bool(((total.double() - dense).abs() <= 1e-5 * size + 1e-12).all())
