"""Rotation of queries and keys 16 bytes at a time (csrc/rope_store.cu): the bits of the kernel that takes a pair at a time."""
import pytest
import torch

DEV = "cuda"


# one item a thread and several, fewer angles than threads and more, part of a head rotated, nothing rotated, no angles
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,kv_heads,d,rotary", [(1, 1, 1, 16, 16), (5, 4, 2, 64, 64), (37, 32, 8, 128, 128), (3, 5, 1, 96, 32), (2, 70, 70, 256, 256),
                                                            (4, 2, 2, 32, 0), (3, 2, 1, 1024, 1024)])
def test_bits_of_a_pair_at_a_time(dtype, tokens, heads, kv_heads, d, rotary):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(tokens + d)
    row = (heads + 2 * kv_heads) * d
    values = torch.randn(tokens, row, generator=gen).to(dtype)
    room = torch.empty(tokens * row + 8, dtype=dtype, device=DEV)
    off = room[1:1 + tokens * row].view(tokens, row)
    off.copy_(values)
    on = values.to(DEV)
    inv_freq = (10000.0 ** (-torch.arange(rotary // 2) / max(1, rotary // 2))).float().to(DEV)
    positions = torch.randint(0, 100000, (tokens,), generator=gen, dtype=torch.int32).to(DEV)
    assert off.data_ptr() % 16 and not on.data_ptr() % 16
    got = ops.rope_store(on, heads, kv_heads, d, inv_freq, rotary, positions)
    want = ops.rope_store(off, heads, kv_heads, d, inv_freq, rotary, positions)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    plain = ops.rope_store(on, heads, kv_heads, d, None, rotary, positions)
    assert torch.equal(torch.cat([p.reshape(tokens, -1) for p in plain], 1), on)
