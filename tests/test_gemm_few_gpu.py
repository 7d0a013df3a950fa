"""bfloat16 products of up to 64 rows with the weights as the wide tcgen05 operand (csrc/gemm_bf16_few.cu), against float64."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# rows around the three tile widths; columns and K that end inside a tile and inside a block of 64; more column tiles than SMs (both
# accumulators); more blocks of K than the ring has stages
@pytest.mark.parametrize("M", [1, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(16, 8), (128, 64), (144, 136), (1040, 520), (3008, 1032), (128 * 150 + 16, 72), (256, 4104)])
@pytest.mark.parametrize("mode", [0, 1, 3])
def test_matches_float64(M, N, K, mode):
    from llama_rs_metal_b200.kernels import gemm_dispatch
    gen = torch.Generator().manual_seed(M + N + K)
    x, w = (torch.randn(rows, K, generator=gen).bfloat16() for rows in (M, N))
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = K * 2.0 ** -23 * size  # a rounding (towards zero) per product added
    shape, dtype = (M, N), torch.float32 if mode == 1 else torch.bfloat16
    if mode == 3:  # |d silu(g) u| <= 1.1 |u| dg + |g| du
        parts, errors = want.view(M, N // 16, 2, 8), bound.view(M, N // 16, 2, 8)
        gate, up = parts[:, :, 0], parts[:, :, 1]
        want = (torch.nn.functional.silu(gate) * up).reshape(M, N // 2)
        bound = (1.1 * up.abs() * errors[:, :, 0] + gate.abs() * errors[:, :, 1]).reshape(M, N // 2) + 2.0 ** -20 * want.abs()
        shape = (M, N // 2)
    if mode != 1:
        bound = bound + 2.0 ** -8 * want.abs()
    out = torch.full(shape, float("nan"), dtype=dtype, device=DEV)
    gemm_dispatch.gemm_bf16_few(x.to(DEV), w.to(DEV), out, mode)
    gemm_dispatch.check_status()
    assert bool(((out.double().cpu() - want).abs() <= bound + 1e-30).all())


@pytest.mark.parametrize("M,N,K", [(13, 19200, 1600), (16, 9480, 3200), (32, 49408, 2048)])
def test_the_rule_takes_it_and_agrees_with_the_other_kernels(monkeypatch, M, N, K):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    assert gemm_dispatch.few_takes(M, N, K, 0)
    gen = torch.Generator(device=DEV).manual_seed(M)
    x, w = (torch.randn(rows, K, generator=gen, device=DEV).bfloat16() for rows in (M, N))
    got = ops.linear(x, w).double()
    monkeypatch.setattr(gemm_dispatch, "umma_width", 128)
    other = ops.linear(x, w).double()
    # both round a float32 sum to bfloat16: at most one step of it apart, and the sums' own difference
    assert bool(((got - other).abs() <= 2.0 ** -7 * other.abs() + K * 2.0 ** -22 * (x.double().abs() @ w.double().abs().T)).all())


# columns for which tiles of fewer than 128 weight rows are taken: 64, 80, 96 and 112 of them, the last one ragged
@pytest.mark.parametrize("N", [9472, 11600, 14032, 16384, 16528])
@pytest.mark.parametrize("M,mode", [(13, 0), (29, 3), (50, 1), (64, 3)])
def test_tiles_of_fewer_rows(N, M, mode):
    test_matches_float64(M, N, 136, mode)
