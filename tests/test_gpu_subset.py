"""The subset test around its work items' edges: queries per item (they set how
many tiles a warp selects for at once), tiles per item, and candidates per
tile around a pass (32), a double pass (64) and a trip (4)."""
import numpy as np
import pytest

from oracle import oracle
from tagmatch_b200 import TagMatch, workload
from tagmatch_b200.tagmatch import filter_from_bits
from tests.helpers import assert_same_multisets

pytestmark = pytest.mark.gpu


def _check(f, ko, k, q, max_p, seg_tiles):
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.set_tiles_per_item(seg_tiles)
        tm.add_many(f, ko, k)
        tm.consolidate(max_p, 1)
        off, keys = tm.match_batch(q)
    eoff, ekeys = oracle.match(f, ko, k, q)
    assert_same_multisets(off, keys, eoff, ekeys)


@pytest.mark.parametrize("nq", [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1500])
@pytest.mark.parametrize("seg_tiles", [1, 37, 128])
def test_queries_per_item(nq, seg_tiles):
    f, ko, k = workload.generate_filters(2500, 61)
    q = workload.generate_queries(nq, f, 61)
    q[0] = q[-1] = 0xFFFFFFFF
    _check(f, ko, k, q, 65536, seg_tiles)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 96, 97, 129])
@pytest.mark.parametrize("nf", [1, 2, 31, 32])
def test_candidates_per_tile(n, nf):
    """One tile of nf filters that share bit 0; n of 700 queries hold it,
    spread over the chunks, and match every second filter."""
    f = np.stack([filter_from_bits([0] + ([10 + i] if i else []) + ([50] if i & 1 else [])) for i in range(nf)])
    ko = np.arange(nf + 1, dtype=np.uint32)
    k = np.arange(nf, dtype=np.uint32)
    q = np.tile(filter_from_bits([1] + list(range(10, 45))), (700, 1))
    at = np.linspace(0, 699, n).astype(int)
    q[at, 0] |= 1
    q[at[::3], 1] |= np.uint32(1 << (50 - 32))
    _check(f, ko, k, q, 65536, 128)


def test_more_records_than_expected():
    """Queries that match every filter make more hit records than the buffer is
    made for at first: the batch runs again and is exact."""
    import torch

    from tagmatch_b200.tagmatch import read_device
    f, ko, k = workload.generate_filters(200_000, 62)
    nq = 300
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add_many(f, ko, k)
        tm.consolidate(65536, 1)
        dq = torch.full((nq, 6), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        for retries in (1, 1):  # the second call finds the buffer grown
            po, pk, nk = tm.match_batch_device(dq.data_ptr(), nq)
            assert tm.match_stats()["pair_retries"] == retries
            assert np.array_equal(read_device(po, nq + 1, np.uint64), np.arange(nq + 1, dtype=np.uint64) * k.size)
        last = read_device(pk + 4 * (nq - 1) * k.size, k.size, np.uint32)
        assert np.array_equal(np.sort(last), np.sort(k))
