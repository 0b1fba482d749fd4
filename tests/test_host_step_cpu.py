"""The host's side of a step: pages handed out many at a time are those that one at a time would have been, a full pool takes
none, and token ids in any numeric form are packed alike."""
import numpy as np
import pytest

import torch

from kindi_b200.cache.pages import CacheFull, FreeList, PageMap
from kindi_b200.cache.sequence_cache import SequenceCache
from kindi_b200.engine.batch import StepEntry, pack
from kindi_b200.kernels import lib as K
from kindi_b200.parts.base import KVNeed


def test_many_ids_at_a_time_are_the_ones_taken_one_by_one():
    a, b = FreeList(9, "page"), FreeList(9, "page")
    for f in (a, b):
        for i in [f.take() for _ in range(6)][1::2]:
            f.give(i)
    assert a.take_many(4) == [b.take() for _ in range(4)]
    a.check()
    left = a.n_free
    with pytest.raises(CacheFull):
        a.take_many(left + 1)
    assert a.n_free == left
    assert a.take_many(0) == []
    a.check()


def test_a_full_pool_leaves_a_sequence_as_it_was():
    pm = PageMap(n_pages=3, n_slots=2)
    pm.ensure(0, 65)
    pm.take_dirty()
    with pytest.raises(CacheFull):
        pm.ensure(1, 129)
    assert pm.take_dirty() == [] and pm.rows[1] == {} and pm.n_blocks[1] == 0
    pm.ensure(0, 10)                                   # nothing new
    assert pm.take_dirty() == []
    pm.ensure(1, 64)
    pm.check()


@pytest.mark.parametrize("form", [tuple, list, lambda t: np.array(t, dtype=np.int64), lambda t: tuple(np.int32(x) for x in t),
                                  lambda t: tuple(float(x) for x in t)])
def test_token_ids_in_any_form(form):
    toks = (3, 0, 70000, 9)
    ps = pack([StepEntry(0, form(toks), (3,)), StepEntry(1, form((5, 6)), ())], [0, 2])
    a, n = ps.off["tok"]
    assert ps.meta[a:a + n].tolist() == [3, 0, 70000, 9, 5, 6]


@pytest.mark.parametrize("toks,want", [
    (bytearray([1, 2, 3, 4]), [1, 2, 3, 4]), (memoryview(bytes([7, 0, 9])), [7, 0, 9]), (np.array([5, 2 ** 31 + 3, 1]), [5, 3 - 2 ** 31, 1]),
    (np.array([[4, 5]], dtype=np.uint8)[0], [4, 5]), (range(3, 6), [3, 4, 5])])
def test_token_ids_that_are_no_tuple_keep_numpys_rules(toks, want):
    """bytes are numbers, and an id beyond 32 bits in an array wraps around to one that the device reports"""
    ps = pack([StepEntry(0, toks, ()), StepEntry(1, (8, 9), ())], [0, 0])
    a, n = ps.off["tok"]
    assert ps.meta[a:a + n].tolist() == want + [8, 9]


def test_ids_beyond_32_bits_in_a_tuple_are_refused():
    with pytest.raises(OverflowError):
        pack([StepEntry(0, (1, 2 ** 31), ())], [0])


class _Event:
    """stands in for the event behind the kernels that read the staging memory"""

    def __init__(self):
        self.recorded = self.waited = 0

    def record(self):
        self.recorded += 1

    def synchronize(self):
        self.waited += 1


def test_staging_memory_is_kept_until_the_kernels_have_read_it():
    cache = SequenceCache([KVNeed(1, 8, None)], max_tokens=128, n_slots=1, dtype=torch.float32, device="cpu")
    event = cache._stage_free = _Event()
    del cache
    assert event.waited == 1


def test_a_failed_launch_leaves_the_launches_before_it_waited_for(monkeypatch):
    cache = SequenceCache([KVNeed(1, 8, None), KVNeed(2, 8, None)], max_tokens=128, n_slots=1, dtype=torch.float32, device="cpu")
    stage, event, calls = torch.zeros(8, 2, dtype=torch.int32), _Event(), []

    def table_set(table, entries, n):
        calls.append(n)
        if len(calls) == 2:
            raise K.KernelError("no")
    monkeypatch.setattr(K, "table_set", table_set)
    cache.device, cache._stage, cache._stage_np, cache._stage_free = torch.device("cuda"), lambda n: stage, stage.numpy(), event
    cache.reserve(cache.alloc_slot(), 100)
    with pytest.raises(K.KernelError):
        cache.flush()
    assert calls == [2, 2] and event.recorded == 1


def test_a_table_of_more_places_than_32_bits_is_written_the_general_way(monkeypatch):
    cache = SequenceCache([KVNeed(1, 8, None)], max_tokens=256, n_slots=2, dtype=torch.float32, device="cpu")
    cache.device = torch.device("cuda")                      # (the table stays where it is)
    monkeypatch.setattr(K, "table_set", lambda *a: pytest.fail("staged"))
    monkeypatch.setattr(SequenceCache, "STAGED_PLACES", 7, raising=False)
    monkeypatch.setattr(SequenceCache, "_stage", lambda self, n: pytest.fail("staged"))
    slots = [cache.alloc_slot() for _ in range(2)]
    for s in slots:
        cache.reserve(s, 100)
    cache.flush()
    table = cache.groups[0].table
    for s in slots:
        assert table[s].tolist() == [cache.groups[0].pages.rows[s].get(b, -1) for b in range(4)]
