"""Bulk adds merged on several threads: the same database, byte for byte, as
the merge with staged single adds, with groups of equal filters (one of them
longer than a thread's stretch), filters without keys and repeated keys."""
import numpy as np
import pytest

from tagmatch_b200 import TagMatch, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4095, 8192, 60_000])
def test_threads_and_staged_merge_agree(tmp_path, n):
    rng = np.random.default_rng(81)
    base = workload.generate_filters(max(1, n // 3), 81)[0]
    f = base[rng.integers(0, base.shape[0], size=n)]
    f[: n // 2] = base[0]  # one group over several stretches
    f = f[rng.permutation(n)]
    counts = rng.integers(0, 5, size=n)
    ko = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    k = rng.integers(0, 50_000, size=int(ko[-1])).astype(np.uint32)
    files = []
    for staged in (False, True):
        db = tmp_path / f"db{int(staged)}"
        with TagMatch() as tm:
            tm.set_database_filename(db)
            half = n // 2
            tm.add_many(f[:half], ko[: half + 1], k[: ko[half]])
            tm.add_many(f[half:], ko[half:], k)  # offsets that do not begin at 0
            if staged:  # one single add of what is there already takes the other merge
                i = int(np.argmax(counts)) if counts.max() else 0
                tm.add(f[i], k[ko[i]: ko[i + 1]])
            tm.consolidate(1000, 1)
        files.append(db.read_bytes())
    assert files[0] == files[1]
