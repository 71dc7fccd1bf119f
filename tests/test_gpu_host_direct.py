"""Host calls into pinned memory on both sides of the batch size (2^24 keys) up
to which keys travel as 32-bit values instead of narrowed ones."""
import ctypes

import numpy as np
import pytest

from tagmatch_b200 import TagMatch, _native
from tagmatch_b200.tagmatch import filter_from_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 16_777, 16_778])
@pytest.mark.parametrize("unique", [False, True])
def test_pinned_results_around_the_direct_limit(nq, unique):
    import torch
    keys = np.arange(1, 65_000, 65, dtype=np.uint32)[:1000]
    q = np.tile(filter_from_bits([3, 9]), (nq, 1))
    with TagMatch() as tm:
        tm.set_persistence(False)
        tm.add(filter_from_bits([3]), keys)
        tm.consolidate(65536, 1)
        off = torch.zeros(nq + 1, dtype=torch.int64).pin_memory()
        out = torch.zeros(nq * 1000 + 8, dtype=torch.int32).pin_memory()
        dq = torch.from_numpy(q.view(np.int32)).pin_memory()
        got = ctypes.c_uint64(0)
        for _ in range(2):
            out.fill_(-1)
            st = _native.load().tm_match_batch(
                tm._h, ctypes.cast(dq.data_ptr(), _native.u32p), nq, int(unique), ctypes.cast(off.data_ptr(), _native.u64p),
                ctypes.cast(out.data_ptr(), _native.u32p), out.numel(), ctypes.byref(got))
            assert st == 0 and got.value == nq * 1000
            assert np.array_equal(off.numpy(), np.arange(nq + 1) * 1000)
            assert np.array_equal(out.numpy()[: nq * 1000].view(np.uint32).reshape(nq, 1000), np.tile(keys, (nq, 1)))
            assert (out.numpy()[nq * 1000:] == -1).all()
