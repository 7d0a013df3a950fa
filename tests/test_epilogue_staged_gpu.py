"""The epilogues of the tcgen05 products (csrc/gemm_epilogue.cuh): rows that reach memory through shared memory, and the SiLU
gate's quotients, against float64."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


def product(x, w, mode, tile, out):
    from llama_rs_metal_b200.kernels import gemm_dispatch, library
    from llama_rs_metal_b200.kernels.ops import _ptr, _stream
    (M, K), N = x.shape, w.shape[0]
    lib, status = library.load(), _ptr(gemm_dispatch._status_word(x.device))
    gemm_dispatch.mark_status_dirty()
    if tile == "pair":
        code = lib.lrm_gemm_bf16_umma_pair(_ptr(x), _ptr(w), _ptr(out), M, N, K, mode, status, _stream())
    else:
        code = lib.lrm_gemm_bf16_umma_rows(_ptr(x), _ptr(w), _ptr(out), M, M, N, K, mode, tile, 1, status, _stream())
    assert code == 0
    gemm_dispatch.check_status()


# rows that end inside a warp's 32 and inside a tile; columns that end inside a piece of 32, on rows with and without 16-byte pitches;
# more tiles than SMs
@pytest.mark.parametrize("tile", [0, 1, 2, 3, "pair"])
@pytest.mark.parametrize("M,N", [(1, 16), (31, 272), (97, 240), (129, 1008), (300, 28704), (65, 203), (65, 206)])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_rows_and_columns_that_end_inside(tile, M, N, mode):
    if mode == 3 and N % 16:
        pytest.skip("gate and up columns alternate in blocks of 8")
    gen = torch.Generator().manual_seed(M + N)
    K = 72
    x, w = (torch.randn(rows, K, generator=gen).bfloat16() for rows in (M, N))
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = K * 2.0 ** -23 * size  # a rounding (towards zero) per product added
    if mode == 3:  # |d silu(g) u| <= 1.1 |u| dg + |g| du
        parts, errors = want.view(M, N // 16, 2, 8), bound.view(M, N // 16, 2, 8)
        gate, up = parts[:, :, 0], parts[:, :, 1]
        want = (torch.nn.functional.silu(gate) * up).reshape(M, N // 2)
        bound = (1.1 * up.abs() * errors[:, :, 0] + gate.abs() * errors[:, :, 1]).reshape(M, N // 2) + 2.0 ** -20 * want.abs()
    if mode in (0, 3):
        bound = bound + 2.0 ** -8 * want.abs()
    guard = 64  # behind the result: nothing may be written there
    flat = torch.full((want.numel() + guard,), 3.0, dtype=torch.float32 if mode in (1, 2) else torch.bfloat16, device=DEV)
    if mode == 2:
        want, bound = want + 3.0, bound + 2.0 ** -23 * (want.abs() + 3.0)
    product(x.to(DEV), w.to(DEV), mode, tile, flat)
    got = flat[:want.numel()].view(want.shape).double().cpu()
    assert bool(((got - want).abs() <= bound + 1e-30).all())
    assert bool((flat[want.numel():] == 3.0).all())


@pytest.mark.parametrize("tile", [1, "pair"])
def test_gate_values_far_out(tile):
    """Both sides of the lines at which the quotient takes another form, and beyond every range; alone and among others."""
    inf, nan = float("inf"), float("nan")
    special = [0.0, 1e-38, -1e-38, 79.5, -79.5, 80.0, -80.0, 80.5, -80.5, -88.5, -89.0, -104.0, 1e4, -1e4, 3e38, -3e38, inf, -inf, nan]
    gates = torch.tensor(special + [0.125 * i - 6 for i in range(96 - len(special))], dtype=torch.float64).bfloat16()
    gates = torch.cat([gates, torch.linspace(-9, 9, 160).bfloat16()])  # 256: pieces without a special value too
    ups = torch.linspace(0.5, 2.0, 256).bfloat16()
    w = torch.zeros(512, 64, dtype=torch.bfloat16)
    w.view(32, 2, 8, 64)[:, 0, :, 0] = gates.view(32, 8)
    w.view(32, 2, 8, 64)[:, 1, :, 0] = ups.view(32, 8)
    x = torch.zeros(70, 64, dtype=torch.bfloat16)
    x[:, 0] = 1.0
    out = torch.zeros(70, 256, dtype=torch.bfloat16, device=DEV)
    product(x.to(DEV), w.to(DEV), 3, tile, out)
    g = gates.double()
    want = (g / (1 + torch.exp(-g)) * ups.double()).expand(70, 256)
    got = out.double().cpu()
    # a rounding to bfloat16; float32 has no more than 2^-149 of the smallest, and over 3.4e38 is infinite either way
    same = (got == want) | (got.isnan() & want.isnan()) | ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-37)
    same |= (want.abs() > 3.39e38) & got.isinf() & (got.sign() == want.sign())
    assert bool(same.all())
