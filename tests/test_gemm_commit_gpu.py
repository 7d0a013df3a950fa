"""Short products of many tiles whose epilogue is the slow part: every tile's accumulator has to reach it, every time."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [128, 192, 256, 512, "pair", "wide"])
def test_every_tile_reaches_the_epilogue(monkeypatch, tile):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    if tile in ("pair", "wide") and gemm_dispatch.pair_room() == 0:
        pytest.skip("no clusters of two CTAs here")
    if tile != "wide":
        monkeypatch.setattr(gemm_dispatch, "umma_width", tile)
    M, N, K = 700, 40000, 72
    gen = torch.Generator(device=DEV).manual_seed(0)
    x, w = (torch.randn(n, K, generator=gen, device=DEV).bfloat16() for n in (M, N))
    want, before = (x.double() @ w.double().T).float(), torch.randn(M, N, generator=gen, device=DEV)
    for rep in range(60):  # 128 x 192 tiles lost one in one of 20 launches
        out = before.clone()
        torch.cuda.synchronize()
        if tile == "wide":
            gemm_dispatch.gemm_bf16_wide(x, w, out, 2, 192)
        else:
            ops.linear(x, w, epilogue=ops.ADD, out=out)
        # K roundings of sums below the largest, and one of the addition
        assert float((out - before - want).abs().max()) <= (K + 2) * 2.0 ** -23 * float(want.abs().max() + before.abs().max()), f"launch {rep}"
    gemm_dispatch.check_status()
