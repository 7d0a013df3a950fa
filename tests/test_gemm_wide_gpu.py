"""bfloat16 products of more than 64 rows with the weights as the wide operand on pairs of SMs (csrc/gemm_bf16_wide.cu)."""
import pytest
import torch

DEV = "cuda"


# rows around whole tiles; columns and K that end inside a tile, inside a CTA's half of it and inside a block of 64; more tiles than
# pairs of SMs (both accumulators); more blocks of K than the ring has stages
@pytest.mark.gpu
@pytest.mark.parametrize("rows", [64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("M,N,K", [(65, 16, 8), (256, 256, 64), (97, 272, 136), (529, 1040, 520), (66, 256 * 75 + 16, 72), (333, 400, 4104)])
@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4])
def test_matches_float64(rows, M, N, K, mode):
    from llama_rs_metal_b200.kernels import gemm_dispatch, library
    gen = torch.Generator().manual_seed(M + N + K)
    x, w = (torch.randn(n, K, generator=gen).bfloat16() for n in (M, N))
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = K * 2.0 ** -23 * size  # a rounding (towards zero) per product added
    slices = library.load().lrm_gemm_bf16_wide_slices(K, 3) if mode == 4 else 1
    shape, dtype = (M, N), torch.bfloat16 if mode in (0, 3) else torch.float32
    before = torch.randn(M, N, generator=gen)
    if mode == 2:
        want = want + before.double()
        bound = bound + 2.0 ** -24 * want.abs()
    if mode == 3:  # |d silu(g) u| <= 1.1 |u| dg + |g| du
        parts, errors = want.view(M, N // 16, 2, 8), bound.view(M, N // 16, 2, 8)
        gate, up = parts[:, :, 0], parts[:, :, 1]
        want = (torch.nn.functional.silu(gate) * up).reshape(M, N // 2)
        bound = (1.1 * up.abs() * errors[:, :, 0] + gate.abs() * errors[:, :, 1]).reshape(M, N // 2) + 2.0 ** -20 * want.abs()
        shape = (M, N // 2)
    if mode in (0, 3):
        bound = bound + 2.0 ** -8 * want.abs()
    out = before.to(DEV) if mode == 2 else torch.full((slices, *shape) if mode == 4 else shape, float("nan"), dtype=dtype, device=DEV)
    gemm_dispatch.gemm_bf16_wide(x.to(DEV), w.to(DEV), out, mode, rows, slices)
    gemm_dispatch.check_status()
    got = out.double().cpu().sum(0) if mode == 4 else out.double().cpu()
    assert bool(((got - want).abs() <= bound + 1e-30).all())


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(70, 3072, 2048), (200, 4096, 4096), (333, 2050, 1032), (529, 2048, 8192)])
def test_the_rule_takes_it_and_agrees_with_the_other_kernels(monkeypatch, M, N, K):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    if gemm_dispatch.pair_room() == 0:
        pytest.skip("no clusters of two CTAs here")
    assert gemm_dispatch.wide_plan(M, N, K, 0, gemm_dispatch.pair_room()) is not None
    gen = torch.Generator(device=DEV).manual_seed(M)
    x, w = (torch.randn(n, K, generator=gen, device=DEV).bfloat16() for n in (M, N))
    got, planes = ops.linear(x, w).double(), gemm_dispatch.gemm_bf16_slices(x, w)
    monkeypatch.setattr(gemm_dispatch, "no_wide", True)
    other, size = ops.linear(x, w).double(), x.double().abs() @ w.double().abs().T
    # both round a float32 sum to bfloat16: at most one step of it apart, and the sums' own difference
    assert bool(((got - other).abs() <= 2.0 ** -7 * other.abs() + K * 2.0 ** -22 * size).all())
    if planes is not None:
        assert bool(((planes.double().sum(0) - other).abs() <= 2.0 ** -8 * other.abs() + K * 2.0 ** -22 * size).all())


def test_the_rule():
    from llama_rs_metal_b200.kernels.gemm_dispatch import WIDE_BLOCK, wide_plan
    for M in (65, 100, 128, 200, 333, 529, 700, 1024, 1500, 2048, 5000):
        for N, K in ((3072, 2048), (2048, 8192), (28672, 4096), (520, 1000), (130, 64)):
            for mode in (0, 1, 2, 3):
                plan = wide_plan(M, N, K, mode, 74)
                if plan is not None:
                    k_blocks = -(-K // 64)
                    assert plan[0] in WIDE_BLOCK and 1 <= plan[1] <= (8 if mode == 2 else 1)
                    assert plan[1] == 1 or (plan[1] - 1) * -(-k_blocks // plan[1]) < k_blocks  # no slice is empty
    # both kernels were timed at these sizes
    faster = [(128, 3072, 2048, 0), (529, 3072, 2048, 0), (128, 6144, 4096, 0), (1024, 6144, 4096, 0), (180, 16384, 2048, 3), (529, 28672, 4096, 3),
              (600, 4096, 14336, 1), (1280, 4096, 14336, 1), (2500, 2048, 2048, 1)]
    slower = [(1024, 28672, 4096, 3), (2048, 4096, 14336, 1), (1500, 3072, 2048, 0), (2048, 16384, 3072, 3)]
    assert all(wide_plan(*sizes, 74) for sizes in faster) and not any(wide_plan(*sizes, 74) for sizes in slower)
