"""Token rows 16 bytes at a time (csrc/embedding.cu): the same numbers as one by one."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
# widths of whole pieces and not, one and several CTAs a row, rows off 16 bytes
@pytest.mark.parametrize("hidden", [1, 4, 8, 12, 24, 250, 1000, 2048, 2056, 3072, 8200])
@pytest.mark.parametrize("scale", [None, 0.37])
@pytest.mark.parametrize("offset", [0, 1])
def test_rows(dtype, hidden, scale, offset):
    from llama_rs_metal_b200.kernels import ops
    vocab = 37
    flat = torch.randn(vocab * hidden + offset, generator=torch.Generator().manual_seed(hidden)).to(dtype).to(DEV)
    table = flat[offset:].view(vocab, hidden)
    ids = torch.tensor([0, vocab - 1, 5, -1, vocab, 5, 17], dtype=torch.int32, device=DEV)
    want = table.float()[ids.clamp(0, vocab - 1).long()] * (1.0 if scale is None else torch.tensor(scale, device=DEV))
    want[3:5] = 0
    assert torch.equal(ops.embed_rows(table, ids, scale), want)
