"""The partitioner's peeled range around what one CTA takes (65,536 filters),
against the oracle's restatement of the reference partitioner: same sets and
masks, and a table built from them that matches as the oracle does."""
import numpy as np
import pytest

from oracle import oracle
from tagmatch_b200 import TagMatch, workload
from tagmatch_b200.tagmatch import balanced_partitioning
from tests.helpers import assert_same_multisets, groups_from_assignment

pytestmark = pytest.mark.gpu


def _filters(n, seed, with_zero):
    f = workload.generate_filters(n, seed)[0]
    if with_zero:
        f[n // 2] = 0
    return f


def _check(f, max_p):
    part, masks, sizes = balanced_partitioning(f, max_p)
    want = oracle.partition(f, max_p)
    assert groups_from_assignment(part, len(sizes)) == sorted(want)
    assert sorted(map(tuple, masks.tolist())) == sorted(tuple(m.tolist()) for m in oracle.masks_of(f, want))
    assert np.array_equal(np.bincount(part, minlength=len(sizes)), sizes)


@pytest.mark.parametrize("n,max_p,with_zero", [(1, 10, True), (2, 10, False), (33, 100, True), (1000, 2000, False),
                                               (1025, 65536, True), (65_535, 65536, False), (65_536, 65536, True),
                                               (65_537, 100_000, False), (90_000, 100_000, True), (200_000, 70_000, False),
                                               (200_000, 1000, True)])
def test_partition_sets(n, max_p, with_zero):
    f = _filters(n, 71, with_zero)
    _check(f, max_p)


def test_one_bit_per_filter():
    """192 peels: filters with one bit each, some more frequent than others
    by a second bit."""
    f = np.zeros((192 * 2, 6), dtype=np.uint32)
    for b in range(192):
        f[2 * b, b >> 5] = 1 << (b & 31)
        f[2 * b + 1, b >> 5] |= np.uint32(1 << (b & 31))
        c = (b + 1) % 192
        f[2 * b + 1, c >> 5] |= np.uint32(1 << (c & 31))
    _check(f, 1000)


@pytest.mark.parametrize("n,max_p", [(50_000, 65536), (150_000, 100_000)])
def test_table_with_peeled_tiles(n, max_p):
    f, ko, k = workload.generate_filters(n, 72)
    q = workload.generate_queries(300, f, 72)
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add_many(f, ko, k)
        tm.consolidate(max_p, 1)
        off, keys = tm.match_batch(q)
    eoff, ekeys = oracle.match(f, ko, k, q)
    assert_same_multisets(off, keys, eoff, ekeys)


@pytest.mark.parametrize("n", [32, 33, 64, 1023, 1024, 1025, 2049, 5000])
@pytest.mark.parametrize("shared_bit", [False, True])
def test_table_around_one_warp_ranges(n, shared_bit):
    """Tile ranges around what one warp splits to its end (1,024 filters); a bit
    that all filters share keeps them in one partition."""
    f, ko, k = workload.generate_filters(n, 73)
    if shared_bit:
        f = np.unique(f | np.array([1, 0, 0, 0, 0, 0], dtype=np.uint32), axis=0)
        ko, k = ko[: f.shape[0] + 1], k[: ko[f.shape[0]]]
    q = workload.generate_queries(200, f, 73)
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add_many(f, ko, k)
        tm.consolidate(65536, 1)
        off, keys = tm.match_batch(q)
    eoff, ekeys = oracle.match(f, ko, k, q)
    assert_same_multisets(off, keys, eoff, ekeys)
