"""Which prompts have their experts sorted where the products go through pairs of SMs (ops.moe_prefers_pairs). No GPU needed."""
import pytest


# (tokens, width, inner width, experts, chosen); both ways were timed at these sizes
@pytest.mark.parametrize("sizes,sorted_", [((256, 2048, 1024, 8, 2), True), ((384, 2048, 1024, 16, 4), True), ((768, 2048, 1024, 8, 4), True),
                                           ((96, 1024, 2048, 16, 4), True), ((1500, 1024, 512, 4, 1), True), ((320, 4096, 1024, 16, 4), True),
                                           ((160, 2048, 1024, 8, 2), False), ((320, 2048, 1024, 8, 4), False), ((384, 1024, 512, 4, 1), False),
                                           ((4096, 768, 384, 16, 8), False), ((200, 4096, 1024, 16, 4), False), ((64, 1024, 2048, 32, 8), False),
                                           ((2048, 512, 256, 4, 1), False), ((500, 72, 40, 8, 2), False)])
def test_the_line(sizes, sorted_):
    from llama_rs_metal_b200.kernels import ops
    assert ops.moe_prefers_pairs(*sizes) is sorted_
