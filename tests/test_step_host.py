"""A step's host side: which token ids are accepted, and a page table that follows the steps without the host waiting for them."""
import numpy as np
import pytest
import torch

from llama_rs_metal_b200.cache import Cache
from llama_rs_metal_b200.engine import StepEntry, validate_entries
from llama_rs_metal_b200.errors import InvalidError
from llama_rs_metal_b200.parts.base import KeyValueRequest


def one_by_one(tokens, vocab):
    for t in tokens:
        if not 0 <= int(t) < vocab:
            return InvalidError
    return None


@pytest.mark.parametrize("tokens", [
    [0, 9], [10], [-1, 3], [3, 10], (1, 2, 3), range(5), [True, 2], [2.9, 9.99], [10.5], [-0.5], [np.int64(4), 5], np.arange(10),
    np.arange(11), np.array([3, 4], dtype=np.uint8), np.array([1.5]), torch.arange(4), torch.arange(12), [2 ** 70], [-2 ** 70],
    [2 ** 63, 1], np.array([2 ** 63], dtype=np.uint64), ["7"], ["x"], [None], [float("nan")], [[1, 2], [3]], np.arange(4).reshape(2, 2)])
def test_tokens_are_taken_and_refused_as_one_by_one(tokens):
    def outcome(fn):
        try:
            return fn()
        except Exception as e:  # noqa: BLE001
            return type(e)
    want = outcome(lambda: one_by_one(tokens, 10))
    assert outcome(lambda: validate_entries([StepEntry(0, tokens)], 10)) is want


@pytest.mark.gpu
def test_page_table_follows_without_waiting_for_the_device():
    cache = Cache([KeyValueRequest(kv_heads=1, head_dim=32)], torch.float32, torch.device("cuda"), 64 * 64, 8, 64 * 8)
    group = cache.kv_groups[0]
    slots = [cache.open_slot() for _ in range(8)]
    streams = [torch.cuda.current_stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    seen, want, waited = [], [], []
    for i in range(24):  # tables taken while the device is busy, on two streams by turns
        with torch.cuda.stream(streams[i // 3 % 2]):
            if i % 3 == 0:
                torch.cuda._sleep(2_000_000)  # about a millisecond
            cache.grow([(slots[i % 8], 64 * (1 + i // 8))])
            cache.commit([(slots[i % 8], 64 * (1 + i // 8))])
            cache.sync()
            seen.append(group.table_device.clone())
            want.append(group.table_host.copy())
            waited.append(streams[i // 3 % 2].query())
    torch.cuda.synchronize()
    assert not all(waited)  # the host went on ahead
    for i, (a, b) in enumerate(zip(seen, want)):
        assert np.array_equal(a.cpu().numpy(), b), f"table {i}"
