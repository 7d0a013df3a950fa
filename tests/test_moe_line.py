"""Which prompts have their experts sorted where the products go through pairs of SMs (ops.moe_prefers_pairs). No GPU needed."""
import pytest


# (tokens, width, inner width, experts, chosen); both ways were timed at these sizes
@pytest.mark.parametrize("sizes,sorted_", [((96, 2048, 1024, 8, 2), True), ((64, 1024, 512, 16, 4), True), ((2048, 2048, 1024, 8, 4), True),
                                           ((64, 1024, 2048, 32, 8), True), ((1024, 1024, 512, 4, 1), True), ((512, 768, 384, 16, 8), True),
                                           ((4096, 768, 384, 16, 8), False), ((160, 2048, 1024, 4, 1), False), ((384, 1024, 512, 4, 1), False),
                                           ((384, 4096, 1024, 8, 4), False), ((2048, 512, 256, 4, 1), False), ((500, 72, 40, 8, 2), False)])
def test_the_line(sizes, sorted_):
    from llama_rs_metal_b200.kernels import ops
    assert ops.moe_prefers_pairs(*sizes) is sorted_


def test_what_one_sm_tiles_gained_by_stays():
    from llama_rs_metal_b200.kernels import ops
    grid = [(t, w, f, e, k) for t in (64, 500, 1500, 4096) for w, f in ((512, 256), (1024, 512), (2048, 1024)) for e, k in ((3, 1), (8, 2), (8, 3), (32, 8))]
    assert all(ops.moe_prefers_pairs(*sizes) for sizes in grid if ops.moe_prefers_sorted(*sizes))
