"""Under the launch profile (kernels/profile.py) the experts' kernels are launched, and timed, one by one: the same bits."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,apart", [
    (7, {"lrm_moe_router", "lrm_moe_experts_grouped"}),
    (600, {"lrm_moe_router", "lrm_moe_sort", "lrm_moe_gather", "lrm_gemm_bf16_wide_experts_gated", "lrm_gemm_bf16_wide_experts", "lrm_moe_combine"})])
def test_experts_one_by_one(monkeypatch, tokens, apart):
    from llama_rs_metal_b200.kernels import gemm_dispatch, library, profile
    from llama_rs_metal_b200.parts.moe import MixtureOfExperts
    from llama_rs_metal_b200.runtime import Runtime
    if not gemm_dispatch.sorted_on_pairs():
        pytest.skip("no clusters of two CTAs here")
    width, ff, experts, top = 1024, 512, 8, 2
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    tensors = {"router.weight": torch.randn(experts, width, generator=gen, device=DEV) * 0.05}
    for e in range(experts):
        for name, shape in (("gate_proj", (ff, width)), ("up_proj", (ff, width)), ("down_proj", (width, ff))):
            tensors["experts.%d.%s.weight" % (e, name)] = (torch.randn(*shape, generator=gen, device=DEV) * 0.05).bfloat16()
    part = MixtureOfExperts(width, ff, experts, top, router_bias=False)
    part.bind(tensors, Runtime(torch.device(DEV), torch.bfloat16))
    x = torch.randn(tokens, width, generator=gen, device=DEV).bfloat16()
    want = part.forward(x, None, None).clone()
    plain = library.load()
    monkeypatch.setattr(profile, "enabled", True)
    monkeypatch.setattr(library, "_library", profile.ProfiledLibrary(plain))
    monkeypatch.setattr(profile, "_rows", {})
    got = part.forward(x, None, None)
    gemm_dispatch.check_status()
    names = {name for name, _ in profile._rows}
    assert apart <= names and not {"lrm_moe_rows_step", "lrm_moe_sorted_step"} & names
    assert torch.equal(got, want)
