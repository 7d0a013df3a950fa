"""Weights that a decode step reads once leave L2 first (no GPU needed): what attention reads of a short context would go in their place."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama_rs_metal_b200", "csrc")


def test_weights_of_few_rows():
    with open(os.path.join(CSRC, "gemm_bf16_few.cu")) as handle:
        source = handle.read()
    calls = re.findall(r"(tma_load_2d\w*)\([^;]*?&(map_\w)", source)
    assert len(calls) == 4 and all((name == "tma_load_2d_once") == (tensor == "map_w") for name, tensor in calls)
