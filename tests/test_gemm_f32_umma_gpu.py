"""float32 products on the tensor cores (csrc/gemm_f32_umma.cu) against float64: rows around its tiles and the kernel for few, matrices off
its tiles of 128 rows and blocks of 64 of K, with one to four slices of K."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"

MATRICES = [(512, 1024), (520, 1032), (1000, 2056), (1537, 4096), (12416, 1088)]  # slices: 2, 2, 4, 4, 1
ROWS = [1, 16, 17, 32, 33, 47, 128, 129, 257]


def _randn(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def _bound(x, w):
    """Four large truncated additions a block at 2^-22 each, as many times seven of the small products at 2^-7 of that (over all blocks,
    in the K 2^-30), and a rounding of 2^-24 for each of the K / 64 additions between blocks."""
    K = x.shape[1]
    return (5 * 2.0 ** -22 + K * 2.0 ** -30) * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("N,K", MATRICES)
@pytest.mark.parametrize("M", ROWS)
def test_products_match_float64_and_a_row_does_not_depend_on_the_batch(M, N, K):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    assert gemm_dispatch.f32_takes_umma(N, K)
    x, w = _randn(M, K), _randn(N, K, seed=1)
    got = ops.linear(x, w)
    assert bool(((got.double() - x.double() @ w.double().T).abs() <= _bound(x, w)).all())
    for r in {0, M // 2, M - 1}:
        assert torch.equal(ops.linear(x[r:r + 1].contiguous(), w)[0], got[r])
    total = _randn(M, N, seed=2)
    want = total + got
    assert torch.equal(ops.linear(x, w, epilogue=ops.ADD, out=total), want)
    gemm_dispatch.check_status()


@pytest.mark.parametrize("T", [5, 40])
def test_grouped_inputs_match_single_ones(T):
    from llama_rs_metal_b200.kernels import ops
    x, w = _randn(3, T, 1024), _randn(2 * 384 + 200, 1024, seed=1)
    got = ops.linear_grouped(x, w, 384)
    for i, (begin, end) in enumerate(((0, 384), (384, 768), (768, 968))):
        want = x[i].double() @ w[begin:end].double().T
        assert bool(((got[:, begin:end].double() - want).abs() <= _bound(x[i], w[begin:end])).all())


@pytest.mark.parametrize("M", [20, 140])
def test_numbers_out_of_the_parts_range(M):
    """Infinities, NaNs and numbers of 2^32 and more are added with float32 FMAs, in their row and column alone; the smallest numbers
    keep their bits."""
    from llama_rs_metal_b200.kernels import ops
    x, w = _randn(M, 1024), _randn(640, 1024, seed=1)
    clean = ops.linear(x, w)
    x[3, 100], x[5, 7], x[6, 1023], x[M - 1, 512] = float("inf"), float("nan"), 3e38, 2.0 ** 41
    w[2, 9], w[600, 64] = float("-inf"), 1e30
    x[8] *= 2.0 ** -118
    got, want = ops.linear(x, w), x.double() @ w.double().T
    rows = torch.tensor([r for r in range(M) if r not in (3, 5, 6, 8, M - 1)], device=DEV)
    cols = torch.tensor([c for c in range(640) if c not in (2, 600)], device=DEV)
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])
    single = want.float()                                    # what float32 can hold
    assert torch.equal(got.isnan(), single.isnan()) and torch.equal(got.isinf(), single.isinf())
    assert torch.equal(got[got.isinf()], single[got.isinf()])
    whole = single.isfinite()
    x[5, 7], x[3, 100], w[2, 9] = 0.0, 0.0, 0.0
    bound = 1024 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1024 * 2.0 ** -149  # a rounding per FMA, and of the smallest
    assert bool(((got.double() - want).abs() <= bound)[whole].all())


# slices of K: 4, 2, 1; numbers beyond the range in the first slice, in the last and in two, where the weights are zero or not
@pytest.mark.parametrize("N,K", [(1000, 2056), (512, 1024), (12416, 1088)])
def test_a_row_out_of_range_does_not_depend_on_the_batch(N, K):
    from llama_rs_metal_b200.kernels import ops
    x, w = _randn(140, K, seed=3), _randn(N, K, seed=4)
    x[0, 5] = x[1, K - 3] = x[2, 9] = x[2, K // 2 + 40] = 2.0 ** 41
    x[3, 70] = float("inf")
    w[::2, 5] = w[::2, K - 3] = w[::2, 9] = 0.0
    w[7, K - 1] = 2.0 ** 50
    got = ops.linear(x, w)
    for rows in (1, 5, 20, 33):
        few = ops.linear(x[:rows].contiguous(), w)
        assert torch.equal(few.isnan(), got[:rows].isnan()) and torch.equal(few.nan_to_num(), got[:rows].nan_to_num())


def test_long_sums_of_large_numbers_stay_in_range():
    """Numbers below 2^40 whose products, brought back, float32 holds, over so long a K in one slice that the sum of the scaled ones was infinite."""
    from llama_rs_metal_b200.kernels import ops
    N, K, number = 12288, 81920, 2.0 ** 39.9
    got = ops.linear(torch.full((2, K), number, device=DEV), torch.full((1, 1), number, device=DEV).expand(N, K).contiguous())
    want = K * torch.tensor(number).double().item() ** 2
    assert bool(((got.double() - want).abs() <= K * 2.0 ** -24 * want).all())  # a rounding per FMA


# one slice of K, two and four; rows cut in the kernel and ahead of it
@pytest.mark.parametrize("N,K", [(12416, 2048), (1537, 1088), (512, 2048), (600, 8192)])
@pytest.mark.parametrize("M", [30, 140])
@pytest.mark.parametrize("numbers", [1, 2, 3, 4, 8, 20, None])
def test_rows_of_few_numbers_are_no_further_off_than_with_fmas(monkeypatch, M, N, K, numbers):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    gen = torch.Generator(device=DEV).manual_seed(K + N)
    x, w = _randn(M, K, seed=5), _randn(N, K, seed=6)
    if numbers is not None:
        x *= torch.rand((M, K), generator=gen, device=DEV).argsort(1) < numbers
    want, got = x.double() @ w.double().T, ops.linear(x, w)
    monkeypatch.setattr(gemm_dispatch, "force_tiled", True)
    other = ops.linear(x, w)
    off, other_off = float((got.double() - want).norm()), float((other.double() - want).norm())
    assert off <= 1.02 * other_off  # (the spread of so many roundings' sum is under 1 %)
    if numbers == 1:  # one rounding, the three low products left out (2^-34) and the small ones' truncated sum (2^-31)
        assert bool(((got.double() - want).abs() <= (2.0 ** -24 + 2.0 ** -30) * want.abs()).all())


def test_rows_off_16_bytes_go_to_the_other_kernels():
    from llama_rs_metal_b200.kernels import ops
    room = torch.empty(9 * 1024 + 1, device=DEV)
    x, w = room[1:].view(9, 1024).copy_(_randn(9, 1024)), _randn(512, 1024, seed=1)
    assert bool(((ops.linear(x, w).double() - x.double() @ w.double().T).abs() <= 1024 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())
