"""Cache index on the GPU (through the C ABI) against the oracle and the golden vectors:
slots, found masks, valid counts, enumeration order and the complete state including the
LRU counters must be bit-exact."""
import threading

import numpy as np
import pytest
import torch

from .conftest import GOLDEN
from .test_oracle_pins import replay

pytestmark = pytest.mark.gpu


class GpuIndexAdapter:
    """EmbCacheLib.IndexCache with numpy in/out, so that the golden replay reads like the
    reference's own usage (CPU tensors in, CPU tensors out)."""

    def __init__(self, cache_size, mode):
        from hades_b200 import EmbCacheLib

        self.ix = EmbCacheLib.IndexCache(cache_size, f"t{id(self)}", True, False, lookup_mode=mode)

    def add(self, ids):
        return self.ix.add(torch.from_numpy(np.ascontiguousarray(ids))).numpy()

    def lookup(self, ids):
        return self.ix.lookup(torch.from_numpy(np.ascontiguousarray(ids))).numpy()

    def reset(self, ids):
        self.ix.reset(torch.from_numpy(np.ascontiguousarray(ids)))

    def get_valid_entries_num(self):
        return self.ix.get_valid_entries_num()

    def getall(self, n):
        a, b = self.ix.getall(n)
        return a.numpy(), b.numpy()


def _eq(a, b, where):
    a, b = np.asarray(a), np.asarray(b)
    assert a.shape == b.shape, where
    bad = np.nonzero(a != b)[0]
    assert bad.size == 0, (where, bad[:5], a[bad[:5]], b[bad[:5]])


@pytest.mark.parametrize("mode", [0, 1])
def test_golden_replay(cuda_lib, mode):
    golden = np.load(GOLDEN / "index_golden.npz")
    for i in range(int(golden["num_scenarios"])):
        ix = GpuIndexAdapter(int(golden[f"s{i}_cache_size"]), mode)
        assert ix.ix.get_capacity() == int(golden[f"s{i}_capacity"])
        assert ix.ix.get_size() == int(golden[f"s{i}_capacity"])
        assert ix.ix.get_space() == int(golden[f"s{i}_space"])
        replay(ix, golden, i, _eq)


def test_known_answers(cuda_lib):
    ix = GpuIndexAdapter(30, 0)
    assert ix.add(np.arange(10)).tolist() == [7, 15, 23, 31, 6, 14, 22, 30, 5, 13]
    assert ix.lookup(np.array([0, 1, 4, 5, 8, 9, 11, 40])).tolist() == [7, 15, 6, 14, 5, 13, -1, -1]
    assert ix.add(np.arange(0, 41, 4)).tolist() == [7, 6, 5, 4, 3, 2, 1, 0, 7, 6, -1]


@pytest.mark.parametrize("cache_size,id_range,batch", [(8, 40, 64), (1000, 3000, 5000),
                                                        (100_000, 1_000_000, 65_536)])
def test_state_matches_oracle(cuda_lib, oracle_mod, cache_size, id_range, batch):
    """Random add / lookup / reset rounds with duplicates inside a batch; after every round
    the exported line ids and LRU counters equal the oracle's."""
    rng = np.random.default_rng(cache_size)
    gpu = GpuIndexAdapter(cache_size, 0)
    ora = oracle_mod.OracleIndex(cache_size)
    for step in range(12):
        n = int(rng.integers(1, batch + 1))
        ids = rng.integers(0, id_range, n, dtype=np.int64)
        if step % 3 == 0:
            ids[: n // 4] = ids[0]  # a hot id, many duplicates
        kind = ["add", "lookup", "lookup", "add", "reset", "lookup"][step % 6]
        if kind == "add":
            _eq(gpu.add(ids), ora.add(ids), (step, kind))
        elif kind == "lookup":
            _eq(gpu.lookup(ids), ora.lookup(ids, touch=True), (step, kind))
        else:
            gpu.reset(ids)
            ora.reset(ids)
        gi, gl = gpu.ix.export_state()
        oi, ol = ora.export()
        _eq(gi.cpu().numpy(), oi, (step, kind, "line ids"))
        _eq(gl.cpu().numpy(), ol, (step, kind, "lru"))


@pytest.mark.parametrize("cache_size", [8, 100, 20_000, 300_000])
def test_lookup_modes_agree(cuda_lib, oracle_mod, cache_size):
    """The sorted-view search and the set-associative probe return the same slots and found
    masks as the oracle, for hits, misses, negative ids and an empty index."""
    from hades_b200 import EmbCacheLib

    rng = np.random.default_rng(cache_size + 1)
    ix = EmbCacheLib.IndexCache(cache_size, f"modes{cache_size}", True, False)
    ora = oracle_mod.OracleIndex(cache_size)
    q = torch.from_numpy(rng.integers(0, cache_size * 4, 10_000, dtype=np.int64)).cuda()
    for mode in (0, 1):  # empty index
        locs, found = ix.cuda_lookup_found(q, mode)
        assert (locs == -1).all() and not found.any()
    ids = rng.integers(0, cache_size * 4, cache_size * 2, dtype=np.int64)
    _eq(ix.add(torch.from_numpy(ids)).numpy(), ora.add(ids), "add")
    qn = rng.integers(-5, cache_size * 4, 50_001, dtype=np.int64)
    want = ora.lookup(qn, touch=False)
    for mode in (0, 1):
        locs, found = ix.cuda_lookup_found(torch.from_numpy(qn).cuda(), mode)
        _eq(locs.cpu().numpy(), want, ("mode", mode))
        _eq(found.cpu().numpy(), want >= 0, ("found", mode))
    # the view follows later changes
    ix.reset(torch.from_numpy(ids[:100]))
    ora.reset(ids[:100])
    want = ora.lookup(qn, touch=False)
    locs, _ = ix.cuda_lookup_found(torch.from_numpy(qn).cuda(), 1)
    _eq(locs.cpu().numpy(), want, "after reset")


def test_open_by_name_and_empty_batches(cuda_lib):
    from hades_b200 import EmbCacheLib

    a = EmbCacheLib.IndexCache(64, "shared_name", True, False)
    b = EmbCacheLib.IndexCache(64, "shared_name", False, False)
    a.add(torch.arange(10))
    assert b.get_valid_entries_num() == 10
    assert b.lookup(torch.arange(3)).tolist() == a.lookup(torch.arange(3)).tolist()
    assert a.add(torch.empty(0, dtype=torch.int64)).numel() == 0
    assert a.lookup(torch.empty(0, dtype=torch.int64)).numel() == 0
    a.reset(torch.empty(0, dtype=torch.int64))
    with pytest.raises(RuntimeError):
        EmbCacheLib.IndexCache(64, "never_created", False, False)


@pytest.mark.parametrize("cache_size,id_range,n", [(64, 300, 5000), (20_000, 60_000, 200_000)])
def test_touch_lru_from_runs(cuda_lib, oracle_mod, cache_size, id_range, n):
    """The run-based LRU ageing (grouping taken from the aggregation's sort) leaves the same
    counters as the sequential rule, for batches with heavy duplication and for unique ids."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(cache_size + n)
    ix = E.IndexCache(cache_size, f"runs{cache_size}", True, False)
    ora = oracle_mod.OracleIndex(cache_size)
    seed_ids = rng.integers(0, id_range, cache_size * 2, dtype=np.int64)
    assert np.array_equal(ix.add(torch.from_numpy(seed_ids)).numpy(), ora.add(seed_ids))
    for rnd in range(3):
        q = rng.integers(0, id_range, n, dtype=np.int64)
        q[: n // 3] = q[0]  # one very hot id
        rng.shuffle(q)
        want = ora.lookup(q, touch=True)
        qd = torch.from_numpy(q).cuda()
        locs = ix.cudalookup(qd)
        assert np.array_equal(locs.cpu().numpy(), want)
        g = torch.zeros((n, 4), device="cuda")
        *_, runs = E.cudaUniqueSegSum(qd, g, id_bits=32, sync=False, want_runs=True)
        ix.cuda_touch_lru_runs(locs, runs)
        assert np.array_equal(ix.export_state()[1].cpu().numpy(), ora.export()[1]), rnd
        # unique ids: every position its own run, with a device-side count
        uq = np.unique(rng.integers(0, id_range, n // 4, dtype=np.int64))
        rng.shuffle(uq)
        want = ora.lookup(uq, touch=True)
        padded = np.concatenate([uq, np.full(100, 7, dtype=np.int64)])  # ignored tail
        locs = ix.cudalookup(torch.from_numpy(padded).cuda())
        ix.cuda_touch_lru_runs(locs, None, torch.tensor([uq.size], device="cuda"))
        assert np.array_equal(locs.cpu().numpy()[: uq.size], want)
        assert np.array_equal(ix.export_state()[1].cpu().numpy(), ora.export()[1]), rnd


# one launch of the sort (up to 8,192 ids), the lists of the sets, the sort again for many ids per set
# (more than 16 per set on average); sets with lists of up to 32 ids, longer ones, copies of one id
@pytest.mark.parametrize("n,cache_size,kind", [(4096, 4000, "uniform"), (4097, 4000, "uniform"), (4097, 1000, "uniform"),
                                               (8192, 4000, "uniform"), (8193, 4000, "uniform"), (8193, 4104, "uniform"),
                                               (70_000, 100_000, "uniform"), (70_000, 100_000, "copies"),
                                               (20_000, 80_000, "strided"), (140_000, 800_000, "distinct"),
                                               (9_000, 160, "uniform"), (66_000, 160, "uniform")])
def test_add_and_lookup_of_large_batches(cuda_lib, oracle_mod, n, cache_size, kind):
    rng = np.random.default_rng(n + cache_size)
    gpu = GpuIndexAdapter(cache_size, 0)
    ora = oracle_mod.OracleIndex(cache_size)
    for step in range(3):
        ids = rng.integers(0, 4 * cache_size, n, dtype=np.int64)
        if kind == "copies":
            ids[rng.random(n) < 0.3] = 12345 + step
        elif kind == "strided":
            ids[: n // 2] = rng.integers(0, 40, n // 2) * (cache_size // 8) * 3 + rng.integers(0, 50, n // 2)
        elif kind == "distinct":
            ids = rng.permutation(4 * cache_size)[:n].astype(np.int64)
        ids[rng.integers(4, n, 5)] = -1  # padding
        got, use = gpu.add(ids), ids >= 0
        _eq(got[use], ora.add(ids[use]), (step, "add"))
        assert (got[~use] == -1).all()
        q = rng.integers(0, 4 * cache_size, n, dtype=np.int64)
        q[rng.random(n) < 0.2] = ids[3]
        _eq(gpu.lookup(q), ora.lookup(q), (step, "lookup"))
        got_ids, got_lru = gpu.ix.export_state()
        want_ids, want_lru = ora.export()
        _eq(got_ids.cpu().numpy(), want_ids, (step, "ids"))
        _eq(got_lru.cpu().numpy(), want_lru, (step, "lru"))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 16_383, 32_768, 32_769, 65_537, 98_306])
def test_host_lookups_in_parts(cuda_lib, oracle_mod, n, mode):
    """Host ids are looked up in parts of up to 32,768: slots, line ids and LRU counters at the edges of the
    parts, with a hot id that ages in every part, ids that are strided in memory, and adds between."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(n)
    ix = E.IndexCache(6000, f"parts{n}_{mode}", True, False, lookup_mode=mode)
    ora = oracle_mod.OracleIndex(6000)
    for rnd in range(3):
        new = rng.integers(0, 20_000, n, dtype=np.int64)
        _eq(ix.add(torch.from_numpy(new)).numpy(), ora.add(new), ("add", rnd))
        q = rng.integers(0, 20_000, 2 * n, dtype=np.int64)[::2]
        q[:: 5] = new[-1]
        _eq(ix.lookup(torch.from_numpy(q)).numpy(), ora.lookup(np.ascontiguousarray(q), touch=True), ("lookup", rnd))
        ids, lru = ix.export_state()
        oi, ol = ora.export()
        _eq(ids.cpu().numpy(), oi, ("line ids", rnd))
        _eq(lru.cpu().numpy(), ol, ("lru", rnd))


@pytest.mark.parametrize("what,n", [("add", 20_000), ("add", 70_000), ("touch", 20_000), ("lookup", 20_000)])
def test_first_call_may_be_captured(cuda_lib, oracle_mod, what, n):
    """A call on a fresh index inside a stream capture: nothing is allocated on first use."""
    from hades_b200 import EmbCacheLib as E
    from hades_b200 import _lib

    rng = np.random.default_rng(2)
    ids = rng.integers(0, 30_000, n, dtype=np.int64)
    ix = E.IndexCache(10_000, f"first_{what}{n}", True, False)
    ora = oracle_mod.OracleIndex(10_000)
    d = torch.from_numpy(ids).cuda()
    if what != "add":
        ora.add(ids[:5000])  # filled without a call that ages or adds
        ix.import_state(*(torch.from_numpy(x) for x in ora.export()))
    lib, st = _lib.load(), torch.cuda.Stream()
    locs = torch.empty_like(d)
    ws = torch.empty(lib.hb_index_add_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        s = _lib.stream_ptr()
        if what == "add":
            _lib.check(lib.hb_index_add(ix.handle, d.data_ptr(), n, locs.data_ptr(), None, ws.data_ptr(), ws.numel(), s))
        elif what == "touch":
            _lib.check(lib.hb_index_lookup(ix.handle, d.data_ptr(), n, locs.data_ptr(), None, 0, s))
            _lib.check(lib.hb_index_touch_lru(ix.handle, locs.data_ptr(), n, ws.data_ptr(), ws.numel(), s))
        else:
            _lib.check(lib.hb_index_lookup_touch(ix.handle, d.data_ptr(), n, locs.data_ptr(), 0, s))
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        want = ora.add(ids) if what == "add" else ora.lookup(ids, touch=True)
        assert np.array_equal(locs.cpu().numpy(), want)
    gi, gl = ix.export_state()
    oi, ol = ora.export()
    assert np.array_equal(gi.cpu().numpy(), oi) and np.array_equal(gl.cpu().numpy(), ol)


def _split_ids(rng, lines, n, low, ids_per_set=6):
    """ids whose sets are [0, lines / 2) (low) or the rest"""
    half = lines // 2
    s = rng.integers(0, half, n) + (0 if low else half)
    return (s + lines * rng.integers(0, ids_per_set, n)).astype(np.int64)


def _load(stream, times=40):
    """Kernels of many blocks, some 50 us each."""
    x = torch.zeros(1 << 26, device="cuda")
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(times):
            x += 1.0
    x.record_stream(stream)


def _same_state(ix, ora, where=None):
    for got, want in zip(ix.export_state(), ora.export()):
        assert np.array_equal(got.cpu().numpy(), want), where


@pytest.mark.parametrize("n", [500, 60_000, 130_000])
def test_what_follows_a_host_lookup_on_another_stream_finds_the_counters_aged(cuda_lib, oracle_mod, n):
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(n)
    ix = E.IndexCache(40_000, f"complete{n}", True, False)
    ora = oracle_mod.OracleIndex(40_000)
    # what is read goes ahead of the kernels that keep the GPU busy, the lookup's own wait behind them
    streams, busy = [torch.cuda.Stream(), torch.cuda.Stream(priority=-1)], torch.cuda.Stream()
    for rnd in range(12):
        new = rng.integers(0, 120_000, 9_000, dtype=np.int64)
        q = rng.integers(0, 120_000, n, dtype=np.int64)
        dnew = torch.from_numpy(new).cuda()
        torch.cuda.synchronize()
        want = ora.lookup(q, touch=True)
        _load(busy)
        with torch.cuda.stream(streams[0]):
            got = ix.lookup(torch.from_numpy(q))
        with torch.cuda.stream(streams[1]):
            _, lru = ix.export_state()
            lru = lru.cpu()
        assert np.array_equal(got.numpy(), want) and np.array_equal(lru.numpy(), ora.export()[1]), rnd
        with torch.cuda.stream(streams[1]):
            got = ix.cuda_add(dnew).cpu().numpy()
        assert np.array_equal(got, ora.add(new)), rnd


@pytest.mark.parametrize("first", ["default", "own"])
@pytest.mark.parametrize("kind", ["touch", "lookup", "add"])
def test_calls_from_two_streams(cuda_lib, oracle_mod, kind, first):
    """Two streams, each with the ids of sets of its own: whichever runs first, the lines are the same."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(7)
    lines = 5000
    ix = E.IndexCache(lines * 8, f"streams_{kind}_{first}", True, False)
    ora = oracle_mod.OracleIndex(lines * 8)
    start = np.concatenate([_split_ids(rng, lines, 30_000, low) for low in (True, False)])
    assert np.array_equal(ix.add(torch.from_numpy(start)).numpy(), ora.add(start))
    streams = [torch.cuda.default_stream() if first == "default" else torch.cuda.Stream(), torch.cuda.Stream()]
    rounds = [[_split_ids(rng, lines, 6000 + 3000 * int(rng.integers(0, 40)), low, 12) for low in (True, False)] for _ in range(20)]
    dev = [[torch.from_numpy(x).cuda() for x in r] for r in rounds]
    locs = [[ix.cudalookup(x) for x in r] for r in dev]
    torch.cuda.synchronize()
    keep = []
    _load(torch.cuda.Stream(), 200)
    for r, l in zip(dev, locs):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                if kind == "touch":
                    ix.cuda_touch_lru(l[k])
                elif kind == "lookup":
                    keep.append(ix.lookup(r[k]))
                else:
                    keep.append(ix.cuda_add(r[k]))
    torch.cuda.synchronize()
    for r in rounds:
        for x in r:
            ora.add(x) if kind == "add" else ora.lookup(x, touch=True)
    _same_state(ix, ora)


@pytest.mark.parametrize("own", [False, True])
def test_ageing_from_two_threads(cuda_lib, oracle_mod, own):
    """Host lookups of several parts in one thread, ageing of slots in another, each of sets of its own, on one
    stream or (own) two."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(8)
    lines = 5000
    ix = E.IndexCache(lines * 8, f"two_threads_{own}", True, False)
    ora = oracle_mod.OracleIndex(lines * 8)
    first = np.concatenate([_split_ids(rng, lines, 30_000, low) for low in (True, False)])
    ix.add(torch.from_numpy(first))
    ora.add(first)
    host = [_split_ids(rng, lines, 120_000, True, 12) for _ in range(10)]
    uniq = [np.unique(_split_ids(rng, lines, 5000, False, 12)) for _ in range(200)]
    slots = [ix.cudalookup(torch.from_numpy(u).cuda()) for u in uniq]
    torch.cuda.synchronize()
    failed, done, enough = [], [], threading.Event()
    _load(torch.cuda.Stream(), 400)

    def touches():
        try:
            with torch.cuda.stream(torch.cuda.Stream() if own else torch.cuda.default_stream()):
                while not enough.is_set():
                    ix.cuda_touch_lru_runs(slots[len(done) % len(slots)], None)
                    done.append(1)
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    t = threading.Thread(target=touches)
    t.start()
    for q in host:
        ix.lookup(torch.from_numpy(q))
    enough.set()
    t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    for q in host + [uniq[k % len(uniq)] for k in range(len(done))]:
        ora.lookup(q, touch=True)
    _same_state(ix, ora)


@pytest.mark.parametrize("n", [786_432, 786_433, 1_000_003])
def test_ageing_of_large_batches(cuda_lib, oracle_mod, n):
    """Marks up to 786,432 positions, sorted by slot beyond; with a hot id and misses.  Without a workspace: marks."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(n)
    ix = E.IndexCache(50_000, f"large{n}", True, False)
    ora = oracle_mod.OracleIndex(50_000)
    first = rng.integers(0, 150_000, 60_000, dtype=np.int64)
    assert np.array_equal(ix.add(torch.from_numpy(first)).numpy(), ora.add(first))
    lib = E._lib.load()
    assert (lib.hb_index_touch_lru_workspace_bytes(n) > 256) == (n > 786_432)
    for rnd in range(3):
        q = rng.integers(0, 150_000, n, dtype=np.int64)
        q[rng.random(n) < 0.2] = first[-1]
        want = ora.lookup(q, touch=True)
        if rnd < 2:
            got = ix.lookup(torch.from_numpy(q) if rnd else torch.from_numpy(q).cuda()).cpu().numpy()
        else:
            locs = ix.cudalookup(torch.from_numpy(q).cuda())
            E._lib.check(lib.hb_index_touch_lru(ix.handle, locs.data_ptr(), n, None, 0, E._lib.stream_ptr()))
            got = locs.cpu().numpy()
        assert np.array_equal(got, want), rnd
        _same_state(ix, ora, rnd)


@pytest.mark.parametrize("n", [1, 31, 32_768, 70_001])
@pytest.mark.parametrize("top", [2**31 - 1, 2**31, 2**40])
def test_host_lookups_of_ids_at_the_edge_of_32_bits(cuda_lib, n, top):
    """A part whose ids fit 32 signed bits crosses PCIe in half the bytes; one with a larger id does not."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(n)
    ix = E.IndexCache(4000, f"edge{n}_{top}", True, False)
    ids = np.concatenate([rng.integers(0, 3000, n, dtype=np.int64), [-1, -2**31, top, top - 1]])[-n:]
    held = torch.from_numpy(np.unique(np.concatenate([np.arange(3000), [2**31 - 2, 2**31 - 1, 2**31, top - 1, top]])))
    ix.cuda_add(held.cuda())
    other = np.where(np.arange(n) % 2 == 0, ids, ids % (1 << 32) if top > 2**31 else ids)  # a low half that is another id
    for q in (ids, other):
        want, _ = ix.cuda_lookup_found(torch.from_numpy(np.ascontiguousarray(q)).cuda())
        _eq(ix.lookup(torch.from_numpy(np.ascontiguousarray(q))).numpy(), want.cpu().numpy(), "slots")


@pytest.mark.parametrize("n,at", [(1, 0), (512, 511), (513, 0), (1025, 511), (1025, 512), (1025, 1023), (40_000, 19_999),
                                  (40_000, 20_000), (40_000, 39_998), (70_001, 30_000)])
def test_host_lookups_with_one_id_beyond_32_bits(cuda_lib, n, at):
    """Parts are narrowed 512 ids at a time until one does not fit; then the part crosses in 64 bits."""
    from hades_b200 import EmbCacheLib as E

    rng = np.random.default_rng(n + at)
    ix = E.IndexCache(4000, f"one_wide{n}_{at}", True, False)
    ids = rng.integers(0, 3000, n, dtype=np.int64)
    ids[at] += 1 << 32  # its low half is an id of the cache
    ix.cuda_add(torch.arange(3000).cuda())
    want, _ = ix.cuda_lookup_found(torch.from_numpy(ids).cuda())
    _eq(ix.lookup(torch.from_numpy(ids)).numpy(), want.cpu().numpy(), "slots")
