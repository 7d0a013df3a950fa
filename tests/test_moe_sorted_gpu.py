"""A prompt's experts on rows sorted by expert (csrc/moe_sorted.cu, gemm_bf16_umma.cu EXPERTS), against float64."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# experts with no pair, one, a whole tile of 128 and one more; more tiles than SMs; N off the column tiles of 256; several
# passes of the sort over the pairs; identity experts
@pytest.mark.parametrize("T,width,ff,E,top,act,identity,skew", [
    (1, 64, 64, 3, 2, 0, 0, False), (128, 128, 64, 4, 1, 1, 0, True), (129, 192, 320, 4, 1, 0, 0, True), (600, 256, 128, 8, 2, 0, 2, False),
    (1500, 512, 192, 16, 4, 1, 0, False), (300, 64, 64, 40, 3, 0, 1, False), (4096, 256, 64, 5, 2, 0, 0, True)])
def test_sorted_rows_match_the_definition_in_float64(T, width, ff, E, top, act, identity, skew):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    gen = torch.Generator().manual_seed(T + width)
    limit, alpha = 0.8, 1.702
    gate_up = (torch.randn(E, 2 * ff, width, generator=gen) / width ** 0.5 * 2).bfloat16()
    down = (torch.randn(width, E, ff, generator=gen) / ff ** 0.5).bfloat16()
    x = torch.randn(T, width, generator=gen).bfloat16()
    score = torch.rand(T, E + identity, generator=gen) + (torch.arange(E + identity) == 0) * (10.0 if skew else 0.0)
    ids = torch.topk(score, top).indices.int()
    weights = torch.rand(T, top, generator=gen)
    want = torch.zeros(T, width, dtype=torch.float64)
    for e in range(E):
        rows = torch.nonzero((ids == e).any(1))[:, 0]
        if rows.numel() == 0:
            continue
        share = (weights.double() * (ids == e)).sum(1)[rows, None]
        both = x[rows].double() @ gate_up[e].double().T
        g, u = both[:, :ff], both[:, ff:]
        if act == ops.ACT_SILU:
            y = torch.nn.functional.silu(g) * u
        else:
            g = g.clamp(max=limit)
            y = g * torch.sigmoid(alpha * g) * (u.clamp(-limit, limit) + 1)
        want[rows] += (share * y) @ down[:, e].double().T
    on = [t.to(DEV) for t in (x, gate_up, down, ids, weights)]
    got = ops.moe_experts_sorted(*on, limit, alpha, act)
    gemm_dispatch.check_status()
    # the gated values are rounded to bfloat16 once (2^-9 each), everything else is float32
    assert float((got.double().cpu() - want).norm() / want.norm().clamp(min=1e-30)) <= 4e-3
    start = torch.randn(T, width, generator=gen)
    added = ops.moe_experts_sorted(*on, limit, alpha, act, out=start.to(DEV))
    assert torch.equal(added, start.to(DEV) + got)
    # the products over all experts, in bfloat16 from the same float32 sums
    every = ops.linear(on[0], on[1].view(E * 2 * ff, width), out_dtype=torch.float32)
    dense = ops.linear(ops.moe_dense_gate(every, on[3], on[4], E, limit, alpha, out_dtype=torch.bfloat16, act=act),
                       on[2].view(width, E * ff), out_dtype=torch.float32)
    assert float((got - dense).norm() / dense.norm().clamp(min=1e-30)) <= 2e-3
