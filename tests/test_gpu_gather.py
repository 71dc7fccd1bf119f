"""The key gather around its steps: runs of keys about 32 (from where the gather
for long runs is taken) and 128 long (from where a batch of 32 runs is copied
one by one), single filters with thousands of keys, and few records spread over
blocks of every size."""
import numpy as np
import pytest

from oracle import oracle
from tagmatch_b200 import TagMatch
from tagmatch_b200.tagmatch import filter_from_bits
from tests.helpers import assert_same_multisets

pytestmark = pytest.mark.gpu


def _check(f, counts, q):
    rng = np.random.default_rng(95)
    ko = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    k = np.concatenate([np.sort(rng.choice(1 << 20, size=c, replace=False)) for c in counts]).astype(np.uint32)
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add_many(f, ko, k)
        tm.consolidate(65536, 1)
        off, keys = tm.match_batch(q)
    assert_same_multisets(off, keys, *oracle.match(f, ko, k, q))


@pytest.mark.parametrize("run", [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 131, 2048])
@pytest.mark.parametrize("nq", [32, 64, 2049])
def test_runs_of_one_length(nq, run):
    """A filter per query, of `run` keys each: every batch is 32 such runs."""
    pairs = [(a, b) for a in range(64) for b in range(a + 1, 64)][:nq if nq < 100 else 200]
    f = np.stack([filter_from_bits(p) for p in pairs])
    q = f[np.arange(nq) % len(pairs)]
    _check(f, [run] * len(pairs), q)


@pytest.mark.parametrize("nq", [1, 63, 65, 500, 2047, 2048, 2049, 10_000])
def test_mixed_runs(nq):
    """Queries over a table in which lengths of 1 to 5,000 lie side by side:
    matches of a few long runs, of many short ones, and of both."""
    lengths = [1, 2, 31, 32, 33, 64, 97, 128, 129, 1000, 2047, 2048, 5000]
    pairs = [(a, b) for a in range(40) for b in range(a + 1, 40)][:300]
    f = np.stack([filter_from_bits(p) for p in pairs])
    counts = [lengths[i % len(lengths)] if i % 3 == 0 else 1 + i % 4 for i in range(len(pairs))]
    rng = np.random.default_rng(nq)
    some = pairs if nq < 3000 else pairs[:60]
    q = np.stack([filter_from_bits(np.concatenate([some[i] for i in rng.integers(0, len(some), size=1 + nq % 2)]))
                  for _ in range(nq)])
    if nq < 3000:
        q[0] = 0xFFFFFFFF  # every filter: many runs in one record
    _check(f, counts, q)
