"""Performance cases of the TagMatch engine: what a program that uses it has it do.

A pub/sub program keeps a table of stored filters (subscriptions as 192-bit
Bloom filters, each with the keys of its subscribers) and matches queries
(messages) against it.  The cases go through the package's public entry
points over the real range: one query to a full device batch, a table of a
quarter million filters to ten million, both result forms (`match` and
`match_unique`), 16-bit and full 32-bit key spaces, even and skewed tag
popularity, large partitions and the API's default ones, device-resident and
host calls, the asynchronous request queue, and building the table.

Tables and queries follow the distributions of csrc/workload.cc (filters of
1-8 Zipf tags over 100,000 tags, 7 bits per tag, 1-4 keys; a query is the
union of 1-3 stored filters and 5-20 more tags, or 10-30 tags), drawn on the
GPU so that a ten-million-filter table takes well under a second to make.

Outputs are whole numbers (offsets and keys, partition ids, masks and sizes)
in buffers that the program keeps from call to call, zero past what a call
writes: device results are copied out of the engine's memory, which the next
call overwrites.  `match` leaves the keys of one query in no particular
order, which may differ from call to call: a case of it returns one query's
keys sorted, and for more queries the offsets (every query's key count).
`match_unique` returns each query's keys in ascending order, so its cases
return offsets and keys as they are.
"""
import ctypes
import math
import threading

import numpy as np
import torch

from tagmatch_b200 import TagMatch, _native
from tagmatch_b200.tagmatch import balanced_partitioning

TAGS = 100_000
HASHES = 7
KEYS16 = 1 << 16
KEYS32 = 1 << 32


def _case(name, entry, filters, queries, unique=True, max_p=65536, tiles=128, zipf=1.0, superset=0.5, keys=KEYS16):
    return {"name": name, "entry": entry, "filters": filters, "queries": queries, "unique": unique, "max_p": max_p,
            "tiles": tiles, "zipf": zipf, "superset": superset, "keys": keys}


def listed():
    return [
        # one message against a table of a million: the latency of the smallest call
        _case("one-query-1m", "device", 1_000_000, 1, unique=False),
        # a serving request of ordinary size against the ten-million table
        _case("request-500-10m", "device", 10_000_000, 500),
        # the throughput headline: a full default device batch (65,536 queries)
        # of plain match on the ten-million table, tiles per item as autotuned
        _case("batch-65536-10m", "device", 10_000_000, 65_536, unique=False, tiles=1024),
        # bulk match_unique, a batch that fills no chunk, work item or warp evenly
        _case("ragged-20011-1m", "device", 1_000_000, 20_011),
        # a table consolidated with the API's default partition size (1,000 filters): thousands of partitions
        _case("default-partitions-4096", "device", 1_000_000, 4_096, max_p=1000),
        # few popular tags and queries that mostly contain stored sets: uneven
        # partitions, dense results
        _case("skewed-8192-2m", "device", 2_000_000, 8_192, zipf=1.3, superset=0.9),
        # keys that are 32-bit ids instead of small ones (the sorting form of match_unique)
        _case("wide-keys-2000", "device", 300_000, 2_000, keys=KEYS32),
        # a serving thread that may not allocate, scratch and outputs fixed
        _case("noalloc-1000", "noalloc", 1_000_000, 1_000),
        # the host call: queries from and results to host memory
        _case("host-3000", "host", 1_000_000, 3_000),
        # continuous serving: a burst of 16 requests of 1-4,096 queries
        # (log-uniform) through the asynchronous queue, results to the host
        _case("burst-16-requests", "submit", 250_000, 16),
        # the partitioner by itself, as a program that lays out its own tables calls it
        _case("partition-1m", "partition", 1_000_003, 0),
        # an update goes live: stage a quarter million filters, consolidate, answer the first queries
        _case("consolidate-250k", "consolidate", 250_000, 256),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["device"] * 6 + ["noalloc", "host", "submit", "partition", "consolidate"])
    case = _case("", entry, log_int(20_000, 4_000_000), 0)
    del case["name"]
    if entry == "partition":
        case["max_p"] = rng.choice([1000, 8192, 65536])
        return case
    case["max_p"] = rng.choice([65536, 65536, 8192, 1000])
    case["zipf"] = rng.choice([1.0, 1.0, 1.3])
    case["superset"] = rng.choice([0.1, 0.5, 0.9])
    case["tiles"] = rng.choice([128, 128, 512, 1024])
    case["queries"] = log_int(1, 40_000)
    if entry == "device":
        case["keys"] = rng.choice([KEYS16, KEYS16, KEYS32])
        case["unique"] = rng.random() < 0.7 and case["queries"] * case["filters"] < 3e10
        if case["keys"] == KEYS32 and case["unique"]:
            # the sorting form holds a query's keys in one block's hands: keep results moderate
            case["filters"] = min(case["filters"], 600_000)
            case["queries"] = min(case["queries"], 8_000)
        elif case["filters"] > 1_000_000:
            case["queries"] = min(case["queries"], 20_000)
    elif entry == "noalloc":
        # all scratch of the call is one 64 MiB array
        case["queries"] = max(1, min(4096, case["queries"], int(6e8 / case["filters"])))
        case["max_p"] = max(case["max_p"], 8192)
    elif entry == "host":
        case["queries"] = min(case["queries"], 10_000, max(1, int(4e9 / case["filters"])))
    elif entry == "submit":
        case["filters"] = min(case["filters"], 600_000)
        case["queries"] = rng.randint(1, 30)
    elif entry == "consolidate":
        case["filters"] = min(case["filters"], 500_000)
        case["queries"] = min(case["queries"], 1024)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _tag_words():
    """[TAGS, 6] words of every tag: 7 bits at splitmix64 positions (csrc/workload.cc)."""
    golden = np.uint64(0x9E3779B97F4A7C15)
    z = np.arange(TAGS, dtype=np.uint64)[:, None] * np.uint64(256) + np.arange(HASHES, dtype=np.uint64) + golden
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    bit = ((z ^ (z >> np.uint64(31))) % np.uint64(192)).astype(np.int64)
    w = np.zeros((TAGS, 6), dtype=np.uint32)
    rows = np.arange(TAGS)
    for i in range(HASHES):
        w[rows, bit[:, i] >> 5] |= np.uint32(1) << (bit[:, i] & 31).astype(np.uint32)
    return torch.from_numpy(w.view(np.int32)).cuda()


class _Draws:
    """Seeded draws on the GPU: Zipf tags and the sets made of them."""

    def __init__(self, seed, zipf):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        self.words = _tag_words()
        p = torch.arange(1, TAGS + 1, dtype=torch.float64, device="cuda") ** -zipf
        self.cdf = torch.cumsum(p, 0) / p.sum()

    def ints(self, n, lo, hi):
        return torch.randint(lo, hi + 1, (n,), generator=self.g, device="cuda")

    def or_tags(self, words, count, most):
        """ORs count[i] Zipf tags into words[i]."""
        n = words.shape[0]
        for t in range(most):
            u = torch.rand(n, dtype=torch.float64, generator=self.g, device="cuda")
            tag = torch.searchsorted(self.cdf, u, right=True).clamp_(max=TAGS - 1)
            words |= torch.where((t < count)[:, None], self.words[tag], torch.zeros((), dtype=torch.int32, device="cuda"))
        return words

    def filters(self, n):
        """n different sets of 1-8 tags, in no order."""
        w = torch.empty((0, 6), dtype=torch.int32, device="cuda")
        while w.shape[0] < n:
            m = int((n - w.shape[0]) * 1.6) + 4096
            more = self.or_tags(torch.zeros((m, 6), dtype=torch.int32, device="cuda"), self.ints(m, 1, 8), 8)
            w = torch.cat([w, more])
            h = torch.zeros(w.shape[0], dtype=torch.int64, device="cuda")
            for k in range(6):
                h = (h ^ (w[:, k].to(torch.int64) & 0xFFFFFFFF)) * -7046029254386353131
                h = h ^ (h >> 29)
            h, at = torch.sort(h, stable=True)
            first = torch.ones_like(h, dtype=torch.bool)
            first[1:] = h[1:] != h[:-1]
            w = w[at[first]]
        return w[:n].contiguous()

    def queries(self, n, stored, superset):
        w = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
        of_stored = torch.rand(n, generator=self.g, device="cuda") < superset
        sets = torch.where(of_stored, self.ints(n, 1, 3), 0)
        for s in range(3):
            pick = stored[self.ints(n, 0, stored.shape[0] - 1)]
            w |= torch.where((s < sets)[:, None], pick, torch.zeros((), dtype=torch.int32, device="cuda"))
        return self.or_tags(w, torch.where(of_stored, self.ints(n, 5, 20), self.ints(n, 10, 30)), 30)


def _host(words):
    return words.cpu().numpy().view(np.uint32)


def _table(d, case):
    """(filters [n, 6], key_offsets [n + 1], keys) on the host, and the filters on the GPU."""
    n = case["filters"]
    f = d.filters(n)
    count = d.ints(n, 1, 4)
    ko = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ko[1:] = torch.cumsum(count, 0)
    keys = torch.randint(0, case["keys"], (int(ko[-1]),), generator=d.g, device="cuda")
    return _host(f), ko.cpu().numpy().astype(np.uint32), keys.cpu().numpy().astype(np.uint32), f


def _engine(case, f, ko, k):
    tm = TagMatch()
    tm.set_persistence(False)
    tm.set_tiles_per_item(case["tiles"])
    tm.add_many(f, ko, k)
    tm.consolidate(case["max_p"], 1)
    return tm


class _DeviceView:
    """Device memory that the engine owns, as torch takes it; keeps the engine alive."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": typestr, "version": 3}


def _view(owner, ptr, count, dtype):
    return torch.as_tensor(_DeviceView(owner, ptr, count, "<i8" if dtype == torch.int64 else "<i4"), device="cuda")


def _request_sizes(count):
    """count request sizes spread log-uniformly over 1 .. 4,096 queries."""
    return [int(round(4096 ** ((i + 0.5) / count))) for i in range(count)]


def _keys_at_most(case):
    """Keys to hold per query: several times the mean of such tables (about 1.5 per 1,000 filters)."""
    return min(case["keys"], 2000 + case["filters"] // (100 if case["queries"] > 16 else 10))


def prepare(case, seed):
    d = _Draws(seed, case["zipf"])
    f, ko, k, stored = _table(d, case)
    entry, nq = case["entry"], case["queries"]
    state = {"case": case}
    if entry == "partition":
        state["filters"] = f
        # ids, masks and sizes of up to `most` partitions
        most = max(4096, case["filters"] // 64)
        state["masks"], state["sizes"] = np.zeros((most, 6), dtype=np.int32), np.zeros(most, dtype=np.int32)
        return state
    sizes = _request_sizes(nq) if entry == "submit" else [nq]
    total = sum(sizes)
    q = d.queries(total, stored, case["superset"])
    room = total * _keys_at_most(case)
    if entry in ("device", "noalloc"):
        state["queries"] = q
        state["stream"] = torch.cuda.Stream()
        state["offsets"] = torch.zeros(nq + 1, dtype=torch.int64, device="cuda")
        if case["unique"] or nq == 1:
            state["keys"] = torch.zeros(room, dtype=torch.int32, device="cuda")
    else:
        # pinned, as a program that calls again and again allocates them
        state["queries"] = q.cpu().pin_memory()
        state["offsets"] = torch.zeros(total + len(sizes), dtype=torch.int64).pin_memory()
        state["keys"] = torch.zeros(room, dtype=torch.int32).pin_memory()
    if entry == "submit":
        state["requests"] = np.split(state["queries"].numpy().view(np.uint32), np.cumsum(sizes)[:-1])
    if entry == "consolidate":
        state["table"] = (f, ko, k)
        return state
    tm = state["tm"] = _engine(case, f, ko, k)
    if entry == "submit":
        tm.set_flush_mode(_native.TM_FLUSH_IMMEDIATE)
        tm.start(4, 1)
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _run_device(state):
    tm, case, n = state["tm"], state["case"], state["case"]["queries"]
    with torch.cuda.stream(state["stream"]):
        po, pk, nk = tm.match_batch_device(state["queries"].data_ptr(), n, unique=case["unique"],
                                           stream=state["stream"].cuda_stream)
        state["offsets"].copy_(_view(tm, po, n + 1, torch.int64))
        if "keys" not in state:
            return state["offsets"]
        if nk:
            keys = _view(tm, pk, nk, torch.int32)
            state["keys"][:nk] = keys if case["unique"] else torch.sort(keys).values
        return state["offsets"], state["keys"]


def _run_noalloc(state):
    tm, nk = state["tm"], ctypes.c_uint64(0)
    tm._check(_native.load().tm_match_batch_device_noalloc(
        tm._h, ctypes.c_void_p(state["queries"].data_ptr()), state["case"]["queries"], 1,
        ctypes.c_void_p(state["offsets"].data_ptr()), ctypes.c_void_p(state["keys"].data_ptr()),
        state["keys"].numel(), ctypes.byref(nk), ctypes.c_void_p(state["stream"].cuda_stream)))
    return state["offsets"], state["keys"]


def _run_host(state, tm):
    nk = ctypes.c_uint64(0)
    tm._check(_native.load().tm_match_batch(
        tm._h, ctypes.cast(state["queries"].data_ptr(), _native.u32p), state["case"]["queries"], 1,
        ctypes.cast(state["offsets"].data_ptr(), _native.u64p), ctypes.cast(state["keys"].data_ptr(), _native.u32p),
        state["keys"].numel(), ctypes.byref(nk)))
    return state["offsets"], state["keys"]


def _run_submit(state):
    tm, requests = state["tm"], state["requests"]
    results, left, done = [None] * len(requests), [len(requests)], threading.Event()
    lock = threading.Lock()

    def taker(i):
        def take(offsets, keys, status):
            results[i] = (offsets.view(np.int64), keys.view(np.int32), status)
            with lock:
                left[0] -= 1
                if not left[0]:
                    done.set()
        return take

    for i, q in enumerate(requests):
        tm.submit(q, taker(i), unique=True)
    done.wait()
    torch.cat([torch.from_numpy(r[0]) for r in results], out=state["offsets"])
    keys = [torch.from_numpy(r[1]) for r in results]
    torch.cat(keys, out=state["keys"][: sum(k.numel() for k in keys)])
    return state["offsets"], state["keys"], [r[2] for r in results]


def run(state):
    entry = state["case"]["entry"]
    if entry == "device":
        return _run_device(state)
    if entry == "noalloc":
        return _run_noalloc(state)
    if entry == "submit":
        return _run_submit(state)
    if entry == "host":
        return _run_host(state, state["tm"])
    if entry == "partition":
        part, masks, sizes = balanced_partitioning(state["filters"], state["case"]["max_p"])
        state["masks"][: len(sizes)] = masks.view(np.int32)
        state["sizes"][: len(sizes)] = sizes.view(np.int32)
        return part.view(np.int32), state["masks"], state["sizes"]
    with _engine(state["case"], *state["table"]) as tm:
        return _run_host(state, tm)


def work(case):
    """The least that a pass moves: queries in, the table's filters once (24
    bytes each), and keys and offsets out.  Keys per query as measured on
    such tables: 1.5 per thousand filters with Zipf 1.0 tags.  The subset
    tests are bitwise, so there are no floating-point operations."""
    n, nq = case["filters"], case["queries"]
    if case["entry"] == "partition":
        return {"bytes": n * 28.0, "flops": 0.0}
    if case["entry"] == "submit":
        nq = sum(_request_sizes(nq))
    keys = n * 1.5e-3
    if case["unique"]:
        keys = case["keys"] * -math.expm1(-keys / case["keys"])
    table = 24.0 * n + (14.0 * n if case["entry"] == "consolidate" else 0.0)
    return {"bytes": table + nq * (24.0 + 8.0 + 4.0 * keys), "flops": 0.0}
