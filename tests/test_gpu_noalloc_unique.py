"""Where the no-allocation match_unique keeps its bitmaps: over the hit records
when they are as long, else in what is left of its 64 MiB array, and when they
fit in neither it sorts.  On both sides of each edge, against the known keys
and the entry point that allocates."""
import ctypes

import numpy as np
import pytest

from tagmatch_b200 import TagMatch, _native
from tagmatch_b200.tagmatch import filter_from_bits, read_device

pytestmark = pytest.mark.gpu


def _check(lists, q, want):
    """lists: (filter, keys) of the table; want: each query's keys, ascending."""
    import torch
    n = q.shape[0]
    off = np.concatenate([[0], np.cumsum([w.size for w in want])]).astype(np.uint64)
    keys = np.concatenate(want)
    with TagMatch() as tm:
        tm.set_persistence(False)
        for f, k in lists:
            tm.add(f, k)
        tm.consolidate(65536, 1)
        dq = torch.from_numpy(np.ascontiguousarray(q).view(np.int32)).cuda()
        torch.cuda.synchronize()
        po, pk, nk = tm.match_batch_device(dq.data_ptr(), n, unique=True)
        assert np.array_equal(read_device(po, n + 1, np.uint64), off) and np.array_equal(read_device(pk, nk, np.uint32), keys)
        d_off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        d_keys = torch.zeros(keys.size + 8, dtype=torch.int32, device="cuda")
        for _ in range(2):  # the second call finds the first one's contents in the array
            d_off.fill_(-1)
            d_keys.fill_(-1)
            torch.cuda.synchronize()
            got = ctypes.c_uint64(0)
            st = _native.load().tm_match_batch_device_noalloc(
                tm._h, ctypes.c_void_p(dq.data_ptr()), n, 1, ctypes.c_void_p(d_off.data_ptr()),
                ctypes.c_void_p(d_keys.data_ptr()), keys.size, ctypes.byref(got), None)
            assert st == 0 and got.value == keys.size
            assert np.array_equal(d_off.cpu().numpy().view(np.uint64), off)
            out = d_keys.cpu().numpy()
            assert np.array_equal(out[: keys.size].view(np.uint32), keys) and (out[keys.size:] == -1).all()


@pytest.mark.parametrize("nq", [1, 682, 683, 1100, 1130, 1138, 1140, 1141, 1142, 1143, 1144, 1146, 1150, 1300, 1500])
def test_bitmaps_larger_than_the_array(nq):
    """Key space 393,216 and 1,600 or 3,190 keys per query: bitmaps of 48 KB, of
    which the array holds some 1,200 beside the keys and the rest."""
    rng = np.random.default_rng(7)
    a, b = (np.unique(np.concatenate([rng.choice(393_216, size=1600, replace=False), e])).astype(np.uint32)
            for e in ([0, 393_215], [5, 70_000]))
    q = np.tile(filter_from_bits([3, 4, 5]), (nq, 1))
    q[1::2] = filter_from_bits([3])
    q[5::100] = 0
    both = np.union1d(a, b)
    want = [np.zeros(0, np.uint32) if i % 100 == 5 else a if i & 1 else both for i in range(nq)]
    _check([(filter_from_bits([3]), a), (filter_from_bits([3, 4]), b)], q, want)


@pytest.mark.parametrize("nq", [2, 31, 1000, 4096])
@pytest.mark.parametrize("missing", [0, 1])
@pytest.mark.parametrize("space", [128, 129])
def test_bitmaps_as_long_as_the_records(nq, missing, space):
    """One tile: a query that matches has one hit record of 16 bytes, as long
    as a bitmap of 128 keys.  The records hold them all exactly, or are short
    by one query without matches, or by the second 16 bytes of larger bitmaps."""
    a, b = np.array([1, 100, space - 1], dtype=np.uint32), np.array([1, 2, 100, 101], dtype=np.uint32)
    q = np.tile(filter_from_bits([3, 4, 5]), (nq, 1))
    if missing:
        q[nq // 2] = 0
    both = np.unique(np.concatenate([a, b]))
    want = [np.zeros(0, np.uint32) if missing and i == nq // 2 else both for i in range(nq)]
    _check([(filter_from_bits([3]), a), (filter_from_bits([3, 4]), b)], q, want)
