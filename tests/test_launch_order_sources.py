"""Kernels that may start before their predecessor ends read what it writes through plain pointers only (no GPU needed).

Loads through `const __restrict__` pointers, and `__ldg`, count as loads of memory that never changes: the compiler may move
them ahead of the wait for the predecessor, and then they read what the predecessor has not written yet."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama_rs_metal_b200", "csrc")

# kernels, and what they may read so: weights and a step's own inputs, which no kernel of the step writes
KERNELS = [
    ("moe_rows.cu", "moe_grouped_kernel", {"W"}),
    ("moe_sorted.cu", "moe_sort_kernel", set()),
    ("moe_sorted.cu", "moe_gather_kernel", set()),
    ("moe_sorted.cu", "moe_sorted_gate_kernel", set()),
    ("moe_sorted.cu", "moe_combine_kernel", set()),
    ("moe.cu", "moe_router_kernel", {"w", "bias", "correction"}),
    ("moe.cu", "moe_dense_gate_wide_kernel", set()),
    ("recurrent_walk.cuh", "walk_prepare_kernel", {"head_decay", "look", "cu_seqlens"}),
    ("attention_decode_cluster.cu", "attention_decode_cluster_kernel",
     {"positions", "inv_freq", "dest_rows", "page_table", "slots", "kv_lens", "order"}),
    ("rope_store.cu", "rope_store_vec_kernel", {"dest_rows", "positions", "inv_freq"}),
    ("embedding.cu", "embed_rows_vec_kernel", {"table"}),
    ("elementwise.cu", "silu_mul_vec_kernel", set()),
    ("elementwise.cu", "add_planes_vec_kernel", set()),
    ("norm.cu", "rms_norm_rows_kernel", {"w"}),
    ("norm.cu", "rms_norm_vec_kernel", {"w", "rows"}),
    ("norm.cu", "rms_norm_cluster_kernel", {"w", "rows"}),
]


@pytest.mark.parametrize("file,kernel,constant", KERNELS, ids=[k for _, k, _ in KERNELS])
def test_results_of_the_predecessor_are_read_through_plain_pointers(file, kernel, constant):
    with open(os.path.join(CSRC, file)) as handle:
        source = handle.read()
    begin = re.search(r"__global__[^;{]*?\b%s\(" % kernel, source).end()
    end = source.index(") {", begin)
    body = source[end:source.index("\n}\n", end)]
    parameters = [" ".join(p.split()) for p in source[begin:end].split(",")]
    held = {p.split()[-1] for p in parameters if p.startswith("const ") and "*" in p and "__restrict__" in p}
    assert "pdl_wait();" in body
    assert held <= constant, f"{kernel}: {sorted(held - constant)}"
    assert len(re.findall(r"__ldg\(", body)) == len(re.findall(r"__ldg\(row \+", body)), f"{kernel}: __ldg of what is not a weight"
