"""A prompt's experts on rows sorted by expert (csrc/moe_sorted.cu, gemm_bf16_umma.cu EXPERTS), against float64."""
import pytest
import torch

DEV = "cuda"
pytestmark = pytest.mark.gpu


# experts with no pair, one, a whole tile of 128 and one more; more tiles than SMs; N off the column tiles of 256; several
# passes of the sort over the pairs; identity experts
@pytest.mark.parametrize("T,width,ff,E,top,act,identity,skew", [
    (1, 64, 64, 3, 2, 0, 0, False), (128, 128, 64, 4, 1, 1, 0, True), (129, 192, 320, 4, 1, 0, 0, True), (600, 256, 128, 8, 2, 0, 2, False),
    (1500, 512, 192, 16, 4, 1, 0, False), (300, 64, 64, 40, 3, 0, 1, False), (4096, 256, 64, 5, 2, 0, 0, True)])
def test_sorted_rows_match_the_definition_in_float64(T, width, ff, E, top, act, identity, skew):
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    gen = torch.Generator().manual_seed(T + width)
    limit, alpha = 0.8, 1.702
    gate_up = (torch.randn(E, 2 * ff, width, generator=gen) / width ** 0.5 * 2).bfloat16()
    down = (torch.randn(width, E, ff, generator=gen) / ff ** 0.5).bfloat16()
    x = torch.randn(T, width, generator=gen).bfloat16()
    score = torch.rand(T, E + identity, generator=gen) + (torch.arange(E + identity) == 0) * (10.0 if skew else 0.0)
    ids = torch.topk(score, top).indices.int()
    weights = torch.rand(T, top, generator=gen)
    want = torch.zeros(T, width, dtype=torch.float64)
    for e in range(E):
        rows = torch.nonzero((ids == e).any(1))[:, 0]
        if rows.numel() == 0:
            continue
        share = (weights.double() * (ids == e)).sum(1)[rows, None]
        both = x[rows].double() @ gate_up[e].double().T
        g, u = both[:, :ff], both[:, ff:]
        if act == ops.ACT_SILU:
            y = torch.nn.functional.silu(g) * u
        else:
            g = g.clamp(max=limit)
            y = g * torch.sigmoid(alpha * g) * (u.clamp(-limit, limit) + 1)
        want[rows] += (share * y) @ down[:, e].double().T
    on = [t.to(DEV) for t in (x, gate_up, down, ids, weights)]
    got = ops.moe_experts_sorted(*on, limit, alpha, act)
    gemm_dispatch.check_status()
    # the gated values are rounded to bfloat16 once (2^-9 each), everything else is float32
    assert float((got.double().cpu() - want).norm() / want.norm().clamp(min=1e-30)) <= 4e-3
    start = torch.randn(T, width, generator=gen)
    added = ops.moe_experts_sorted(*on, limit, alpha, act, out=start.to(DEV))
    assert torch.equal(added, start.to(DEV) + got)
    # the products over all experts, in bfloat16 from the same float32 sums
    every = ops.linear(on[0], on[1].view(E * 2 * ff, width), out_dtype=torch.float32)
    dense = ops.linear(ops.moe_dense_gate(every, on[3], on[4], E, limit, alpha, out_dtype=torch.bfloat16, act=act),
                       on[2].view(width, E * ff), out_dtype=torch.float32)
    assert float((got - dense).norm() / dense.norm().clamp(min=1e-30)) <= 2e-3


@pytest.mark.parametrize("T", [400, 500, 700])  # on both sides of the rule between all experts and sorted rows
@pytest.mark.parametrize("residual,shared,gate,identity,pending", [
    (False, False, False, 0, False), (False, True, False, 0, False), (False, True, True, 2, False), (False, False, False, 2, False),
    (True, False, False, 0, False), (True, True, False, 2, False), (True, True, True, 0, False), (True, False, False, 0, True),
    (True, True, False, 0, True), (True, False, False, 2, False)])
def test_the_part_takes_sorted_rows_and_adds_what_it_should(monkeypatch, T, residual, shared, gate, identity, pending):
    """MixtureOfExperts.forward: onto the stream or by itself, beside a shared part with and without its gate, identity experts
    of the float32 stream, partial sums of the part before still pending (they keep the product over all experts, which folds
    them, unless the shared part has settled them)."""
    from llama_rs_metal_b200.engine.batch import StepContext
    from llama_rs_metal_b200.kernels import gemm_dispatch, ops
    from llama_rs_metal_b200.parts.base import PartSpec
    from llama_rs_metal_b200.parts.moe import MixtureOfExperts
    from llama_rs_metal_b200.runtime import Runtime
    width, ff, inner, E, top = 1024, 512, 64, 8, 2
    gen = torch.Generator().manual_seed(T)
    part = MixtureOfExperts(width, ff, E, top, activation="silu", router_bias=False, scoring="softmax_all" if identity else
                            "softmax_chosen", identity=identity, shared_gate=gate,
                            shared=PartSpec("gated_mlp", dict(hidden_size=width, intermediate_size=inner)) if shared else None)
    w = {name: torch.randn(spec.shape, generator=gen) / spec.shape[-1] ** 0.5 for name, spec in part.tensors().items()}
    w = {name: (t * (3 if "router" in name else 1)).to(DEV).bfloat16() for name, t in w.items()}
    runtime = Runtime(torch.device(DEV), torch.bfloat16)
    part.bind(w, runtime)
    stream = torch.randn(T, width, generator=gen).to(DEV)
    x = stream.bfloat16()
    none = torch.zeros(0, dtype=torch.int32, device=DEV)
    ctx = StepContext(runtime, "prefill", T, 1, T, T, *[none] * 7)
    ctx.stream = stream if identity and not residual else None
    start = torch.randn(T, width, generator=gen).to(DEV)
    planes = torch.randn(2, T, width, generator=gen).to(DEV)
    ctx.pending = planes.clone() if pending else None
    took, plain = [], ops.moe_experts_sorted
    monkeypatch.setattr(ops, "moe_experts_sorted", lambda *a, **k: took.append(plain(*a, **k)) or took[-1])
    got = part.forward(x, ctx, start.clone() if residual else None)
    got = ctx.settle(got) if residual else got
    gemm_dispatch.check_status()
    ids, weights = part.route(x)
    f = {name: t.double() for name, t in w.items()}
    x64, want = x.double(), torch.zeros(T, width, dtype=torch.float64, device=DEV)
    for e in range(E):
        g, u = (x64 @ f[f"experts.{e}.{n}_proj.weight"].T for n in ("gate", "up"))
        share = (weights.double() * (ids == e)).sum(1, keepdim=True)
        want += share * ((torch.nn.functional.silu(g) * u) @ f[f"experts.{e}.down_proj.weight"].T)
    want += (weights.double() * (ids >= E)).sum(1, keepdim=True) * (x64 if ctx.stream is None else stream.double())
    if shared:
        g, u = (x64 @ f[f"shared.{n}_proj.weight"].T for n in ("gate", "up"))
        beside = (torch.nn.functional.silu(g) * u) @ f["shared.down_proj.weight"].T
        want += beside * (torch.sigmoid(x64 @ f["shared.gate"].T) if gate else 1.0)
    base = (start.double() if residual else 0.0) + (planes.double().sum(0) if pending else 0.0)
    # the gated values are rounded to bfloat16 once (2^-9 each), everything else is float32
    assert float((got.double() - base - want).norm() / want.norm()) <= 4e-3
    assert len(took) == (1 if T >= 500 and (shared or not pending) else 0) and all(t is not None for t in took)
