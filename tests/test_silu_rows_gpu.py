"""The SiLU gate 16 bytes at a time (csrc/elementwise.cu) has the bits of the kernel that takes a number at a time."""
import pytest
import torch

DEV = "cuda"


# one piece and several in a block, one block and several in a row, a last CTA that is not full; addresses off 16 bytes keep the other kernel
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,inter,block", [(1, 8, 8), (3, 24, 8), (7, 96, 48), (333, 104, 8), (65, 4096, 4096)])
def test_bits_of_a_number_at_a_time(dtype, rows, inter, block):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(rows + inter)
    room = torch.empty(rows * 2 * inter + 16, dtype=dtype, device=DEV)
    values = (torch.randn(rows, 2 * inter, generator=gen) * 30).to(dtype)
    values[0, 0], values[-1, -1] = float("inf"), float("nan")
    one, other = room[1:1 + values.numel()].view(rows, 2 * inter), values.to(DEV)
    one.copy_(values)
    got, want = ops.silu_mul(other, block), ops.silu_mul(one, block)
    assert one.data_ptr() % 16 and not other.data_ptr() % 16
    assert bool(((got == want) | (got.isnan() & want.isnan())).all())
    parts = values.double().view(rows, inter // block, 2, block)
    g, u = parts[:, :, 0].reshape(rows, inter), parts[:, :, 1].reshape(rows, inter)
    near = (g * torch.sigmoid(g) * u).to(dtype).double()
    # of gates below -88.7 the division's denominator is infinite: what is lost is at most |g| exp(-88.7) |u|
    lost = (g * u).abs().nan_to_num(0.0) * 3.1e-39
    ok = (got.double().cpu() - near).abs() <= (2.0 ** -20 if dtype == torch.float32 else 2.0 ** -7) * near.abs() + lost + 1e-37
    assert bool((ok | ~near.isfinite()).all())
