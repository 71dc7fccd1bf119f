"""match_unique on both sides of where bitmaps give way to sorting (8 M words in
all; 1,024, 2,048 and 4,096 words each; 32 keys, a twentieth and an eighth of
the words per query), bitmaps around one, two and four rounds of a warp, and the warp's sort of up to 32 keys with keys that occur twice."""
import numpy as np
import pytest

from tagmatch_b200 import TagMatch
from tagmatch_b200.tagmatch import filter_from_bits

pytestmark = pytest.mark.gpu


def _check(space, counts, nq):
    """Query kinds i: bits 2i and 2i + 1, which match two filters with counts[i]
    keys in all, a third of them in both; the last kind matches nothing."""
    rng = np.random.default_rng(11)
    lists, kinds, want = [], [], []
    for i, n in enumerate(counts):
        a = np.unique(rng.integers(0, space, size=max(1, n * 2 // 3)))
        b = np.unique(np.concatenate([rng.choice(a, size=min(a.size, n // 3), replace=False),
                                      rng.integers(0, space, size=n - a.size - min(a.size, n // 3)) if n > a.size + n // 3
                                      else np.zeros(0, np.int64)]))
        if i == 0:
            a = np.unique(np.append(a, [0, space - 1]))  # the ends of the space: the largest key sets the route
        lists.append((filter_from_bits([2 * i]), a))
        if b.size:
            lists.append((filter_from_bits([2 * i, 2 * i + 1]), b))
        kinds.append(filter_from_bits([2 * i, 2 * i + 1]))
        want.append(np.union1d(a, b).astype(np.uint32))
    kinds.append(filter_from_bits([191]))
    want.append(np.zeros(0, np.uint32))
    which = np.arange(nq) % len(kinds)
    with TagMatch() as tm:
        tm.set_persistence(False)
        for f, k in lists:
            tm.add(f, k.astype(np.uint32))
        tm.consolidate(65536, 1)
        off, keys = tm.match_batch(np.stack(kinds)[which], unique=True)
    assert np.array_equal(np.diff(off.astype(np.int64)), [want[w].size for w in which])
    assert np.array_equal(keys, np.concatenate([want[w] for w in which]))


@pytest.mark.parametrize("words", [1023, 1024, 2047, 2048, 4095, 4096, 12288, 1 << 27])
@pytest.mark.parametrize("counts", [[1, 2, 3, 5, 8], [30, 31, 32, 33, 34], [60, 100, 31, 32, 1], [100, 120, 140, 150],
                                    [240, 260, 300], [600, 620, 650], [1800, 1850, 1900]])
def test_sides_of_the_rule(words, counts):
    _check(words * 32, counts, 8300)


@pytest.mark.parametrize("words", [1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 257])
def test_bitmap_rounds(words):
    for nq in (100, 700):  # 1,024 threads to mark, and fewer
        _check(words * 32, [1, 31, 200, 3000], nq)


@pytest.mark.parametrize("words", [1024, 2048])
def test_sides_of_the_batch_size(words):
    edge = (8 << 20) // words
    for nq in (edge - 1, edge, edge + 1):
        _check(words * 32, [1, 7, 20], nq)
