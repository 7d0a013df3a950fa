"""The norm of many rows with a warp each, and of rows with and without room to spare in a CTA's registers (csrc/norm.cu)."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [4, 100, 1024, 1028, 2048, 2052, 3072, 4096, 4100, 8192])
@pytest.mark.parametrize("n_rows,planes", [(1, 0), (148, 3), (149, 3), (1023, 0), (1024, 0), (1029, 0), (1029, 2)])
@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
def test_against_float64(hidden, n_rows, planes, w_dtype):
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator().manual_seed(hidden + n_rows)
    x, w = torch.randn(n_rows, hidden, generator=gen), torch.randn(hidden, generator=gen).to(w_dtype)
    parts = torch.randn(planes, n_rows, hidden, generator=gen) if planes else None
    total = x.double() + (parts.double().sum(0) if planes else 0)
    gain = w.double() / (total.square().mean(-1, keepdim=True) + 1e-5).sqrt()
    want = total * gain
    stream = x.to(DEV)
    got = ops.rms_norm(stream, w.to(DEV), 1e-5, torch.bfloat16, partials=parts.to(DEV) if planes else None)
    # a rounding to bfloat16; float32 sums: of the planes beside the total's size, of the squares, and a few roundings more
    size = x.double().abs() + (parts.double().abs().sum(0) if planes else 0)
    bound = 2.0 ** -8 * want.abs() + (planes + 8) * 2.0 ** -23 * (size * gain.abs() + want.abs()) + 1e-30
    assert bool(((got.double().cpu() - want).abs() <= bound).all())
    if planes:
        assert bool(((stream.double().cpu() - total).abs() <= planes * 2.0 ** -23 * size).all())
