"""tm_set_memory_budget holds for what match_unique takes beside the keys."""
import threading

import numpy as np
import pytest

from tagmatch_b200 import TagMatch, _native
from tagmatch_b200.tagmatch import filter_from_bits

pytestmark = pytest.mark.gpu


def test_bitmaps_stay_within_the_budget():
    """60,000 queries of two keys in a key space of 32,000: bitmaps of 4 KB each,
    hundreds of times the keys, 240 MB in one batch.  Two lanes of 64 MB may
    hold 128 MB; the rest of the bound is for the offsets and the allocator's
    granularity."""
    import torch
    torch.cuda.init()
    nq, budget = 60_000, 64 << 20
    keys = np.array([3, 31_999], dtype=np.uint32)
    q = np.tile(filter_from_bits([3, 9]), (nq, 1))
    q[::7] = 0
    got, done = [], threading.Event()
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add(filter_from_bits([3]), keys)
        tm.consolidate(65536, 1)
        tm.match_batch(q[:10], unique=True)
        tm.set_memory_budget(budget)
        tm.set_flush_mode(_native.TM_FLUSH_IMMEDIATE)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        tm.start()
        for _ in range(4):
            done.clear()
            tm.submit(q, lambda off, k, st: (got.append((off, k, st)), done.set()), unique=True)
            assert done.wait(60)
        taken = free - torch.cuda.mem_get_info()[0]
        tm.stop()
    counts = np.where(np.arange(nq) % 7 == 0, 0, 2)
    for off, k, st in got:
        assert st == 0
        assert np.array_equal(np.diff(off.astype(np.int64)), counts)
        assert np.array_equal(k, np.tile(keys, counts.sum() // 2))
    assert taken <= 2 * budget + (32 << 20), taken
