"""The paged cache as a Python object (no GPU; a recorder stands where the binding is called): copies of a cache in use, and rows
counted from the end or out of range."""
import copy
import pickle

import pytest
import torch

from pope_pytorch_b200 import PagedKVCache, kv_cache


class Recorder:
    """In the place of the extension module; its page objects, as the real ones, can be neither copied nor pickled."""

    def __init__(self):
        self.maps, self.appends = [], []

    def Pages(self, *tensors):
        return (lambda: tensors)

    def kv_map(self, pages, index, value):
        self.maps.append((list(index), list(value)))

    def kv_append(self, pages, k, v, row):
        self.appends.append(row)


@pytest.fixture
def ops(monkeypatch):
    recorder = Recorder()
    monkeypatch.setattr(kv_cache.N, "_ops", lambda: recorder)
    return recorder


def make():
    return PagedKVCache(3, 2, 64, num_pages=8, page_size=64, max_seq_len=256, device="cpu")


def rows(n):
    return torch.randn(2, n, 64).bfloat16()


@pytest.mark.parametrize("again", [copy.deepcopy, lambda c: pickle.loads(pickle.dumps(c))])
def test_a_cache_in_use_can_be_copied(ops, again):
    cache = make()
    cache.append_to(1, rows(70), rows(70))
    twin = again(cache)
    assert twin.lens == [0, 70, 0] and twin.alloc.table == cache.alloc.table and twin.alloc is not cache.alloc
    assert twin.k_pages.data_ptr() != cache.k_pages.data_ptr() and torch.equal(twin.k_pages, cache.k_pages)
    twin.append_to(0, rows(1), rows(1))
    assert twin._pages()()[0] is twin.k_pages and cache._pages()()[0] is cache.k_pages
    assert twin.lens == [1, 70, 0] and cache.lens == [0, 70, 0]


def test_negative_rows_count_from_the_end(ops):
    cache = make()
    cache.append_to(-1, rows(70), rows(70))
    assert cache.lens == [0, 0, 70] and ops.maps == [([2 * 4, 2 * 4 + 1], [0, 1])] and ops.appends == [2]
    cache.release(-1)
    assert cache.lens == [0, 0, 0] and ops.maps[1] == ([-3], [0])


@pytest.mark.parametrize("b", [3, -4])
def test_rows_outside_the_cache_change_nothing(ops, b):
    cache = make()
    for call in (lambda: cache.append_to(b, rows(70), rows(70)), lambda: cache.release(b)):
        with pytest.raises(IndexError):
            call()
    assert cache.lens == [0, 0, 0] and len(cache.alloc.free) == 8 and ops.maps == [] and ops.appends == []
