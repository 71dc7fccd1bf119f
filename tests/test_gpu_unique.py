"""match_unique at the sizes where its kernels change course: key spaces at the
edge of a bitmap, results around a warp, a block's shared memory and its
two size classes, digits that all keys share."""
import numpy as np
import pytest

from oracle import oracle
from tagmatch_b200 import TagMatch
from tagmatch_b200.tagmatch import filter_from_bits

pytestmark = pytest.mark.gpu

# keys per query; the sorting route's classes meet at 4,096 and 22,528 keys
COUNTS = [1, 2, 31, 32, 33, 255, 256, 257, 1000, 4095, 4096, 4097, 8191, 22527, 22528, 22529, 60000]


def _table(space, counts, seed):
    """Query i holds bits 2i and 2i + 1 and matches two filters, {2i} and
    {2i, 2i + 1}, that share keys: counts[i] keys in all, drawn from
    [0, space)."""
    rng = np.random.default_rng(seed)
    filters, keys, queries = [], [], []
    for i, n in enumerate(counts):
        m = min(n, space)
        first = rng.choice(space, size=(m + 1) // 2, replace=False) if space <= 1 << 20 else np.unique(
            rng.integers(0, space, size=(m + 1) // 2))
        second = np.concatenate([first[: m // 4], rng.integers(0, space, size=m // 2 - m // 4)])
        filters += [filter_from_bits([2 * i]), filter_from_bits([2 * i, 2 * i + 1])]
        keys += [np.unique(first).astype(np.uint32), np.unique(second).astype(np.uint32)]
        queries.append(filter_from_bits([2 * i, 2 * i + 1]))
    # the largest key of the space is in the table, so it sets the route
    keys[0] = np.unique(np.append(keys[0], np.uint32(space - 1)))
    used = [i for i, k in enumerate(keys) if k.size]
    f = np.stack([filters[i] for i in used])
    ko = np.concatenate([[0], np.cumsum([keys[i].size for i in used])]).astype(np.uint32)
    return f, ko, np.concatenate([keys[i] for i in used]), np.stack(queries)


@pytest.mark.parametrize("space", [1, 32, 33, 4096, 65536, 393_215, 393_216, 393_217, 1 << 24, 1 << 32])
def test_unique_routes(space):
    f, ko, k, q = _table(space, COUNTS, 5)
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add_many(f, ko, k)
        tm.consolidate(65536, 1)
        off, keys = tm.match_batch(q, unique=True)
    eoff, ekeys = oracle.match(f, ko, k, q, unique=True)
    assert np.array_equal(off, eoff)
    assert np.array_equal(keys, ekeys)


def test_unique_shared_digits():
    """Keys that differ in one byte only, each byte in turn: the passes over
    the other bytes move nothing."""
    for shift in (0, 8, 16, 24):
        f = np.stack([filter_from_bits([0]), filter_from_bits([0, 1])])
        base = np.uint64(0x5A5A5A5A) & ~(np.uint64(0xFF) << np.uint64(shift))
        both = [np.unique(base | (np.arange(a, 256, 3, dtype=np.uint64) << np.uint64(shift))).astype(np.uint32) for a in (0, 1)]
        ko = np.array([0, both[0].size, both[0].size + both[1].size], dtype=np.uint32)
        k = np.concatenate(both)
        q = np.stack([filter_from_bits([0, 1]), filter_from_bits([0]), filter_from_bits([5])])
        with TagMatch() as tm:
            tm.set_persistence(False)
            tm.add_many(f, ko, k)
            tm.consolidate(65536, 1)
            off, keys = tm.match_batch(q, unique=True)
        eoff, ekeys = oracle.match(f, ko, k, q, unique=True)
        assert np.array_equal(off, eoff) and np.array_equal(keys, ekeys)


@pytest.mark.parametrize("nq", [131_072, 140_000])
def test_many_queries_with_few_small_keys(nq):
    """16-bit keys on both sides of where the bitmaps of a batch (8 KB per
    query) give way to sorting."""
    import torch

    from tagmatch_b200.tagmatch import read_device
    keys = [np.array([7, 9, 65_535], dtype=np.uint32), np.array([1, 9, 30_000], dtype=np.uint32)]
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add(filter_from_bits([3]), keys[0])
        tm.add(filter_from_bits([3, 4]), keys[1])
        tm.consolidate(65536, 1)
        q = np.tile(filter_from_bits([3, 4, 5]), (nq, 1))
        q[1::2] = filter_from_bits([3])
        q[::1000] = 0
        dq = torch.from_numpy(q.view(np.int32)).cuda()
        torch.cuda.synchronize()
        po, pk, nk = tm.match_batch_device(dq.data_ptr(), nq, unique=True)
        off, got = read_device(po, nq + 1, np.uint64), read_device(pk, nk, np.uint32)
    both = np.array([1, 7, 9, 30_000, 65_535], dtype=np.uint32)
    want = [np.zeros(0, np.uint32) if i % 1000 == 0 else keys[0] if i & 1 else both for i in range(nq)]
    assert np.array_equal(np.diff(off.astype(np.int64)), [w.size for w in want])
    assert np.array_equal(got, np.concatenate(want))
