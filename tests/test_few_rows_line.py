"""Which products of few rows take the weights as the wide operand, and which float32 results are cut (gemm_dispatch). No GPU needed."""
from llama_rs_metal_b200.kernels import gemm_dispatch


def test_gates_of_few_tiles_stream_up_to_eight_rows():
    plan = gemm_dispatch.few_plan
    assert plan(8, 8192, 4096, 3) == plan(8, 9216, 3072, 3) == 0 and plan(9, 8192, 4096, 3) == 1
    assert plan(4, 10240, 4096, 3) == plan(8, 28672, 4096, 3) == 1 and plan(8, 16384, 2048, 3) == 0


def test_results_wanted_at_once_are_cut_where_that_was_the_faster_way():
    cut = gemm_dispatch.cut_plan
    faster = [(8, 4096, 14336), (16, 2048, 8192), (64, 1024, 4096), (32, 3072, 2048), (100, 2048, 8192), (500, 2048, 8192), (300, 4096, 14336)]
    slower = [(8, 4096, 8192), (16, 2048, 2048), (48, 8192, 2048), (32, 2048, 2048), (300, 2048, 2048), (100, 6144, 4096), (2048, 8192, 2048)]
    assert all(cut(*sizes, 74) for sizes in faster) and not any(cut(*sizes, 74) for sizes in slower)


# (rows, columns, K, mode, added): whole decode steps were timed both ways at these sizes, of models of widths between the usual ones too
def test_what_up_to_eight_rows_stream_and_what_not():
    plan = gemm_dispatch.few_plan
    wide = [(1, 19456, 2560, 3), (8, 20480, 2560, 3), (4, 28672, 2048, 3), (8, 17920, 3328, 3), (1, 24576, 2560, 1), (8, 32768, 2048, 1), (1, 128256, 2048, 1),
            (1, 12288, 4096, 0), (1, 2560, 8192, 4, True), (8, 4096, 14336, 4, True), (4, 5120, 5120, 4, True), (8, 6144, 4096, 4), (8, 8192, 6144, 4)]
    streamed = [(1, 18432, 2560, 3), (8, 16384, 2048, 3), (8, 16384, 3072, 3), (1, 2048, 8192, 4, True),
                (8, 4096, 6144, 4, True), (8, 3584, 3584, 4, True), (1, 3840, 3328, 4), (8, 4608, 3584, 4), (8, 5120, 3072, 4)]
    assert all(plan(*sizes) for sizes in wide) and not any(plan(*sizes) for sizes in streamed)
