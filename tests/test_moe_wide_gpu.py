"""A prompt's sorted experts on pairs of SMs with the weights as the wide operand (csrc/gemm_bf16_wide.cu EXPERTS, GATED): beside the
tiles of one SM, and against float64."""
import pytest
import torch

DEV = "cuda"


# ff on and off the 128 gate columns of a pair's tile, widths on and off its 256 rows, one block of K and more than the ring has stages,
# experts without a pair, more tiles than pairs of SMs (both accumulators, both phases of the gates' barriers), no weight
@pytest.mark.gpu
@pytest.mark.parametrize("T,width,ff,E,top,act", [(70, 64, 64, 3, 2, 0), (300, 128, 128, 4, 1, 1), (513, 64, 192, 5, 2, 1), (700, 192, 320, 4, 3, 0),
                                                  (4096, 64, 1024, 8, 2, 1), (1000, 832, 448, 6, 2, 0), (5000, 2048, 64, 3, 1, 1)])
def test_beside_the_other_tiles_and_float64(monkeypatch, T, width, ff, E, top, act):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    if not gemm_dispatch.sorted_on_pairs():
        pytest.skip("no clusters of two CTAs here")
    gen = torch.Generator().manual_seed(T + ff)
    gate_up = (torch.randn(E, 2 * ff, width, generator=gen) * 2 / width ** 0.5).bfloat16().to(DEV)
    down = (torch.randn(width, E, ff, generator=gen) / ff ** 0.5).bfloat16().to(DEV)
    x = torch.randn(T, width, generator=gen).bfloat16().to(DEV)
    score = torch.rand(T, E, generator=gen)
    score[:, 1] = -1.0  # nobody's, unless all are chosen
    ids = torch.topk(score, top).indices.int().to(DEV)
    weights = torch.rand(T, top, generator=gen).to(DEV)
    weights[::7] = 0.0
    got = ops.moe_experts_sorted(x, gate_up, down, ids, weights, 7.0, 1.702, act)
    gemm_dispatch.check_status()
    monkeypatch.setattr(gemm_dispatch, "no_wide", True)
    other = ops.moe_experts_sorted(x, gate_up, down, ids, weights, 7.0, 1.702, act)
    xd, want, size, first = x.double(), torch.zeros(T, width, dtype=torch.float64, device=DEV), 0.0, 0.0
    for e in range(E):
        both, summed = xd @ gate_up[e].double().T, xd.abs() @ gate_up[e].double().abs().T
        g, u = both[:, :ff], both[:, ff:]
        if act == 0:
            g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0) + 1
        weight = (weights.double() * (ids == e)).sum(-1, keepdim=True)
        slope = 1.702 if act == 0 else 1.0
        y = weight * g * torch.sigmoid(slope * g) * u
        # what the first product's sums may be off by (a rounding towards zero per product), through the gate, and y's rounding
        off = width * 2.0 ** -23 * (1.1 * u.abs() * summed[:, :ff] + g.abs() * summed[:, ff:]) * weight + 2.0 ** -8 * y.abs()
        want += y @ down[:, e].double().T
        size = size + y.abs() @ down[:, e].double().abs().T
        first = first + off @ down[:, e].double().abs().T
    bound = first + ff * 2.0 ** -23 * size + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())
    assert bool(((got.double() - other.double()).abs() <= 2 * bound).all())
