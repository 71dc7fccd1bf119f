"""The learned flush mode matches its batches in the work items that the cost
model was asked about: tiles per item as it chose them, which recorded batches
also take as they are."""
import os
import re
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

# Prints, for each candidate number of tiles, the items of a recorded batch of
# the queries, then those of the same queries served in the learned mode.
SCRIPT = """
import sys, threading
import numpy as np
from tagmatch_b200 import TagMatch, _native, workload
f, ko, k = workload.generate_filters(100_000, 91)
q = workload.generate_queries(8192, f, 91)
tm = TagMatch()
tm.set_persistence(False)
tm.add_many(f, ko, k)
tm.consolidate(65536, 1)
tm.sched_record(True)
for seg in (32, 128, 512, 2048, 8192):
    tm.set_tiles_per_item(seg)
    for b in (512, 1000, 8192):
        tm.set_batch_limit(b)
        tm.match_batch(q)
tm.sched_train(epochs=20)
tm.set_batch_limit(65536)
n = 1000
for seg in (32, 64, 128, 256, 512, 1024, 2048, 4096, 8192):
    tm.set_tiles_per_item(seg)
    print("candidate", seg, file=sys.stderr, flush=True)
    tm.match_batch(q[:n])
tm.sched_record(False)
tm.set_tiles_per_item(128)
tm.set_flush_mode(_native.TM_FLUSH_LEARNED)
tm.start()
done = threading.Event()
print("served", file=sys.stderr, flush=True)
tm.submit(q[:n], lambda off, keys, status: done.set())
assert done.wait(60)
tm.stop()
tm.close()
"""


def test_served_items_are_a_candidates():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "TM_WORK_COUNTERS": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
    items, label = {}, None
    for line in r.stderr.splitlines():
        if line.startswith(("candidate", "served")):
            label = line
        m = re.match(r"\[tm work\] queries 1000 .* items (\d+)", line)
        if m and label:
            items[label] = int(m.group(1))
    assert len(items) == 10
    assert items["served"] in [v for label, v in items.items() if label != "served"]
