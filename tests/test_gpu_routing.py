"""Routing and queue filling where they change course: queries around a vote,
a CTA, a queue-filling CTA and a count group; partitions around a vote, a CTA
and a window of the routing matrix."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from tagmatch_b200 import TagMatch, _native, workload
from tagmatch_b200.tagmatch import read_device
from tests.helpers import assert_same_multisets

pytestmark = pytest.mark.gpu


def _engine(f, ko, k, max_p):
    tm = TagMatch()
    tm.set_persistence(False)
    tm.add_many(f, ko, k)
    tm.consolidate(max_p, 1)
    return tm


@pytest.fixture(scope="module")
def table():
    f, ko, k = workload.generate_filters(3000, 41)
    return f, ko, k, workload.generate_queries(24_577, f, 41)


@pytest.mark.parametrize("nq", [1, 31, 32, 33, 255, 257, 2047, 2048, 2049, 8191, 8192, 8193, 16_385, 24_577])
@pytest.mark.parametrize("max_p", [65536, 40])
def test_queries_around_edges(table, nq, max_p):
    f, ko, k, q = table
    # some queries that every partition takes, at the ends
    q = q[:nq].copy()
    q[0] = q[-1] = 0xFFFFFFFF
    with _engine(f, ko, k, max_p) as tm:
        off, keys = tm.match_batch(q)
    eoff, ekeys = oracle.match(f, ko, k, q)
    assert_same_multisets(off, keys, eoff, ekeys)


@pytest.mark.parametrize("n", [31, 32, 33, 63, 64, 65, 127, 129, 1100])
def test_partitions_around_edges(n):
    f, ko, k = workload.generate_filters(n, 43)
    q = workload.generate_queries(700, f, 43)
    with _engine(f, ko, k, 1) as tm:
        assert tm.table_info()["partitions"] >= n
        off, keys = tm.match_batch(q)
    eoff, ekeys = oracle.match(f, ko, k, q)
    assert_same_multisets(off, keys, eoff, ekeys)


def test_routing_matrix_in_windows():
    """40,000 partitions x 16,385 queries: the matrix takes two windows."""
    f, ko, k = workload.generate_filters(40_000, 44)
    q = workload.generate_queries(16_385, f, 44)
    with _engine(f, ko, k, 1) as tm:
        tm.set_batch_limit(32_768)
        off, keys = tm.match_batch(q)
    assert np.array_equal(oracle.digest(off, keys), oracle.match_digest(f, ko, k, q))


def test_no_alloc_routing_windows():
    """Slices that leave the static array too little for the whole matrix."""
    import torch
    f, ko, k = workload.generate_filters(10_380, 45)
    nq = 4096
    q = np.zeros((nq, 6), dtype=np.uint32)  # matches nothing, but for three queries that match everything
    q[[0, 1000, nq - 1]] = 0xFFFFFFFF
    with _engine(f, ko, k, 1) as tm:
        assert 10_300 < tm.table_info()["partitions"] <= 10_400
        dq = torch.from_numpy(q.view(np.int32)).cuda()
        d_off = torch.zeros(nq + 1, dtype=torch.int64, device="cuda")
        d_keys = torch.zeros(3 * k.size + 16, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        got = ctypes.c_uint64(0)
        for _ in range(2):
            st = _native.load().tm_match_batch_device_noalloc(
                tm._h, ctypes.c_void_p(dq.data_ptr()), nq, 0, ctypes.c_void_p(d_off.data_ptr()),
                ctypes.c_void_p(d_keys.data_ptr()), d_keys.numel(), ctypes.byref(got), None)
            assert st == 0, _native.load().tm_last_error(tm._h)
            off = d_off.cpu().numpy().view(np.uint64)
            po, pk, nk = tm.match_batch_device(dq.data_ptr(), nq)
            assert got.value == nk == 3 * k.size
            assert np.array_equal(off, read_device(po, nq + 1, np.uint64))
            assert_same_multisets(off, d_keys.cpu().numpy().view(np.uint32)[:nk], off, read_device(pk, nk, np.uint32))
