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


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,n_rows", [(1024, 1480), (1024, 1481), (2048, 1184), (2048, 1185), (3072, 1100), (4096, 1024), (4096, 1185)])
def test_one_round_of_ctas_keeps_a_row_each(hidden, n_rows):
    """Up to eight rows an SM (ten of short rows) have the bits that a few rows have; beyond, a warp's order of the sum."""
    from llama_rs_metal_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(n_rows)
    x, w = torch.randn(n_rows, hidden, generator=gen, device=DEV), torch.randn(hidden, generator=gen, device=DEV).bfloat16()
    got = ops.rms_norm(x, w, 1e-5, torch.bfloat16)
    few = torch.cat([ops.rms_norm(part.contiguous(), w, 1e-5, torch.bfloat16) for part in x.split(500)])
    assert torch.equal(got, few) == (n_rows <= (1184 if hidden >= 2048 else 1480))
    want = x.double() * (w.double() / (x.double().square().mean(-1, keepdim=True) + 1e-5).sqrt())
    assert bool(((got.double() - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs() + 1e-30).all())
