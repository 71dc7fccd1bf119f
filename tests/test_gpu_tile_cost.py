"""Putting neighbouring tiles together: bits that all filters hold say nothing
about which queries are candidates, so the tiles come out the same with one
such bit or with many (a tag that all filters share sets seven)."""
import numpy as np
import pytest

from oracle import oracle
from tagmatch_b200 import TagMatch, workload
from tests.helpers import assert_same_multisets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 20_000])
def test_shared_bits_leave_the_tiles(n):
    base = workload.generate_filters(n, 74)[0]
    base[:, 5] &= np.uint32((1 << 25) - 1)  # bits 185 .. 191 are no filter's own
    base = np.unique(base, axis=0)
    ko = np.arange(base.shape[0] + 1, dtype=np.uint32)
    k = np.arange(base.shape[0], dtype=np.uint32)
    tiles = []
    for shared in (1, 3, 7):
        f = base.copy()
        f[:, 5] |= np.uint32(((1 << shared) - 1) << 25)
        q = workload.generate_queries(100, f, 74)
        with TagMatch() as tm:
            tm.set_persistence(False)
            tm.add_many(f, ko, k)
            tm.consolidate(65536, 1)
            tiles.append(tm.table_info()["tiles"])
            off, keys = tm.match_batch(q)
        assert_same_multisets(off, keys, *oracle.match(f, ko, k, q))
    assert tiles[0] == tiles[1] == tiles[2]
