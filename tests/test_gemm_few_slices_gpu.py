"""Products of up to 64 rows in K slices on the kernel with the weights as the wide operand, and attention that adds them up."""
import numpy as np
import pytest
import torch

DEV = "cuda"


# K that ends inside a block and inside a slice, one slice, more items than SMs, more blocks of K than the ring has stages
@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 8, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K,slices", [(16, 72, 2), (272, 1032, 5), (3008, 520, 3), (128 * 60, 264, 4), (256, 4104, 3), (130, 200, 1)])
@pytest.mark.parametrize("rows", [0, 48, 128])
def test_planes_add_up(M, N, K, slices, rows):
    from llama_rs_metal_b200.kernels import gemm_dispatch, library
    slices = library.load().lrm_gemm_bf16_few_slices(K, slices)
    gen = torch.Generator().manual_seed(M + N + K)
    x, w = (torch.randn(n, K, generator=gen).bfloat16() for n in (M, N))
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    out = torch.full((slices, M, N), float("nan"), device=DEV)
    gemm_dispatch.gemm_bf16_few(x.to(DEV), w.to(DEV), out, 4, slices, rows)
    gemm_dispatch.check_status()
    assert bool(((out.double().cpu().sum(0) - want).abs() <= K * 2.0 ** -23 * size + 1e-30).all())


@pytest.mark.gpu
@pytest.mark.parametrize("d,Hq,Hk,rotary", [(32, 4, 2, 32), (64, 32, 8, 64), (128, 24, 8, 128), (128, 6, 6, 64), (64, 40, 2, 0)])
@pytest.mark.parametrize("cluster", [1, 2, 5])
@pytest.mark.parametrize("n_planes", [1, 3, 9])
def test_attention_adds_the_planes_up(monkeypatch, d, Hq, Hk, rotary, cluster, n_planes):
    """The same bits as from the sum of the planes, rounded to bfloat16: output and cache."""
    from llama_rs_metal_b200.cache import Cache
    from llama_rs_metal_b200.kernels import attention_dispatch, ops
    from llama_rs_metal_b200.parts.base import KeyValueRequest
    monkeypatch.setattr(attention_dispatch, "force_cluster_size", cluster)
    lengths = [1, 64, 65, 333, 700]
    B, W = len(lengths), (Hq + 2 * Hk) * d
    gen = torch.Generator(device=DEV).manual_seed(d + Hq)
    planes = torch.randn(n_planes, B, W, generator=gen, device=DEV) * n_planes ** -0.5
    whole = planes[0].clone()
    for p in range(1, n_planes):
        whole += planes[p]
    inv_freq = (10000.0 ** (-torch.arange(rotary // 2, dtype=torch.float64) * 2 / rotary)).float().to(DEV) if rotary else None
    outs, kept = [], []
    for qkv in (whole.bfloat16(), planes):
        cache = Cache([KeyValueRequest(Hk, d)], torch.bfloat16, torch.device(DEV), 64 * 64, B, 64 * 16)
        slots = [cache.open_slot() for _ in lengths]
        cache.grow([(s, n) for s, n in zip(slots, lengths)])
        cache.sync()
        view = cache.view(0)
        fill = torch.Generator(device=DEV).manual_seed(1)
        for t in (view.k, view.v):
            t.copy_(torch.randn(t.shape, generator=fill, device=DEV).bfloat16())
        dest = cache.destination_rows(slots, [n - 1 for n in lengths], [1] * B)[0]
        i32 = lambda v: torch.tensor(np.asarray(v), dtype=torch.int32, device=DEV)  # noqa: E731
        outs.append(ops.attention_decode_fused(qkv, Hq, inv_freq, rotary, i32([n - 1 for n in lengths]), view, i32(dest), i32(slots),
                                               i32(lengths), max(lengths), d ** -0.5, i32(np.argsort(-np.array(lengths)))))
        kept.append((view.k.clone(), view.v.clone()))
    assert torch.equal(outs[0], outs[1])
    assert all(torch.equal(a, b) for a, b in zip(*kept))


def test_the_rule():
    from llama_rs_metal_b200.kernels.gemm_dispatch import few_plan
    for M in (1, 8, 9, 16, 33, 64, 65):
        for N, K in ((3072, 2048), (2048, 8192), (6144, 4096), (520, 1000), (130, 64), (32768, 3072)):
            for mode in (0, 1, 3, 4):
                slices = few_plan(M, N, K, mode)
                assert 0 <= slices <= (-(-K // 64) if mode == 4 else 1) and (M <= 64 or slices == 0)
                assert slices <= 1 or (slices - 1) * -(-(-(-K // 64)) // slices) < -(-K // 64)  # no slice is empty
    # whole steps were timed with these either way: narrow products go in slices, what is added behind few rows streams
    assert few_plan(8, 6144, 4096, 4) == 3 and few_plan(64, 3072, 2048, 4) == 6 and few_plan(12, 4096, 14336, 4, added=True) == 4
    assert not few_plan(8, 4096, 4096, 4, added=True) and not few_plan(16, 2048, 2048, 4, added=True) and not few_plan(8, 3072, 2048, 4)
    assert few_plan(1, 32768, 2048, 1) and few_plan(4, 28672, 4096, 3) and not few_plan(4, 16384, 2048, 3) and not few_plan(16, 4096, 4096, 0)
