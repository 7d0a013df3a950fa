"""Products whose float32 result is wanted at once, cut into K slices whose planes a launch adds up (gemm_dispatch.cut_plan)."""
import pytest
import torch

DEV = "cuda"


# both kernels, the fewest and the most rows of each, sizes off the tiles; stored and added to what is there
@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(4, 4096, 14336), (9, 520, 8200), (16, 1024, 6144), (17, 3072, 2048), (33, 257, 2048), (64, 2048, 8192), (64, 1000, 4104),
                                   (65, 2048, 8192), (100, 522, 14344), (129, 1024, 4096), (500, 2048, 8192)])
def test_the_sum_of_the_slices(M, N, K):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    gen = torch.Generator().manual_seed(M + N)
    x, w = torch.randn(M, K, generator=gen).bfloat16().to(DEV), torch.randn(N, K, generator=gen).bfloat16().to(DEV)
    planes = gemm_dispatch.gemm_bf16_cut(x, w)
    assert planes is not None and planes.shape[0] > 1
    begun = torch.randn(M, N, generator=gen).to(DEV)
    stored, added = ops.linear(x, w, out_dtype=torch.float32), ops.linear(x, w, ops.ADD, begun.clone())
    gemm_dispatch.check_status()
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # the tensor cores cut off 2^-23 of a sum for each of a slice's products of 16, then the planes' additions round
    off = (K / 16 + 80) * 2.0 ** -23 * size
    assert bool(((stored.double() - want).abs() <= off).all())
    assert bool(((added.double() - begun.double() - want).abs() <= off + 2.0 ** -23 * begun.double().abs() * 80).all())
    assert torch.equal(ops.linear(x, w, out_dtype=torch.float32), stored)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 4, 1000, 4100])
@pytest.mark.parametrize("count", [1, 7, 8, 9, 20])
def test_planes_are_added_in_their_order(n, count):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(n + count)
    x, planes = torch.randn(n, generator=gen), torch.randn(count, n, generator=gen) * 1e3
    want = x.clone()
    for p in planes:
        want += p
    assert torch.equal(ops.add_planes_(x.to(DEV), planes.to(DEV)).cpu(), want)
