"""A prompt's q|k|v projection apart from its rotation and stores (gemm_dispatch.qkv_apart): the bits of the product that rotates and
stores in its epilogue."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("M,heads,kv_heads,d,K", [(65, 32, 8, 128, 4096), (100, 64, 8, 128, 8192), (333, 24, 8, 128, 3072), (560, 32, 8, 128, 4096),
                                                  (128, 40, 12, 64, 3072)])
def test_the_bits_of_the_epilogue(M, heads, kv_heads, d, K):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    gen = torch.Generator().manual_seed(M)
    N = (heads + 2 * kv_heads) * d
    x, w = torch.randn(M, K, generator=gen).bfloat16().to(DEV), (torch.randn(N, K, generator=gen) * 0.02).bfloat16().to(DEV)
    positions = torch.randint(0, 5000, (M,), generator=gen, dtype=torch.int32).to(DEV)
    inv_freq = (500000.0 ** (-torch.arange(d // 2) / (d // 2))).float().to(DEV)
    if gemm_dispatch.pair_room() > 0:
        assert gemm_dispatch.qkv_apart(M, N, K)
    got = ops.rope_store(ops.linear(x, w), heads, kv_heads, d, inv_freq, d, positions)
    want = ops.linear_rope_store(x, w, heads, kv_heads, d, ops.rope_table(positions, inv_freq))
    gemm_dispatch.check_status()
    assert want is not None and all(torch.equal(a, b) for a, b in zip(got, want))
    assert not any(gemm_dispatch.qkv_apart(*sizes) for sizes in ((64, N, K), (700, N, K), (320, 10240, 8192), (128, 3072, 2048)))
