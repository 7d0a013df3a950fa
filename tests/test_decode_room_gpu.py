"""How many CTAs of decode attention an SM holds (csrc/attention_decode_cluster.cu), which is what the size of its clusters is chosen by."""
import pytest

SM_BYTES, SYSTEM = 228 * 1024, 1024


def by_memory(d, cluster, rows):
    """CTAs an SM's shared memory has room for: the ring of pages, what the cluster's CTAs send one another, and the sines and cosines."""
    stages = {32: 3, 64: 3, 128: 2}[d]
    runs = -(-rows * d // 128)
    sent = cluster * (-(-runs // cluster) * 128 + 32) * 4 if cluster > 1 else 0
    return SM_BYTES // (2 * stages * 64 * (d + 8) * 2 + sent + d * 4 + SYSTEM)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("cluster", range(1, 15))
def test_rows_of_a_head_group_cost_no_room(d, cluster):
    """As many as for a single row wherever ring and messages leave room for as many."""
    import torch
    from llama_rs_metal_b200.kernels import library
    torch.zeros(1, device="cuda")
    room = library.load().lrm_attention_decode_cluster_resident
    for rows in range(2, 17):
        if by_memory(d, cluster, rows) == by_memory(d, cluster, 1):
            assert room(d, cluster, rows) == room(d, cluster, 1), rows


@pytest.mark.gpu
@pytest.mark.parametrize("seqs,kv_heads,group,d,keys,size", [(28, 8, 4, 64, 1000, 2), (32, 8, 4, 64, 1000, 2), (37, 8, 4, 64, 1000, 2),
                                                             (19, 8, 8, 128, 1000, 2), (24, 8, 8, 128, 1000, 2), (27, 8, 8, 128, 1000, 2)])
def test_clusters_of_two_where_four_or_three_ctas_fit(seqs, kv_heads, group, d, keys, size):
    from llama_rs_metal_b200.kernels import attention_dispatch
    assert attention_dispatch.decode_cluster_size(seqs, kv_heads, group, d, keys) == size
