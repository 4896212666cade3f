"""Cold-gradient staging table (insert / accumulate / flush) and the sparse optimiser updates
against the oracle's restatement of python/EmbCache/server.py and sparse_optim.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RTOL = 1e-5


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dim", [3, 64, 128])
def test_cold_cache_rounds(cuda_lib, oracle_mod, mode, dim):
    """Several server iterations: flush, insert uncached rows, accumulate remote and local cold
    gradients.  Ids / counts / slot state bit-exact; rows exact too (every slot receives the
    same fp32 additions in the same order as the oracle)."""
    from hades_b200.cold_cache import ColdCache

    rng = np.random.default_rng(dim * 10 + mode)
    num_nodes, entries, clients, local_nodes = 20_000, 2_000, 4, 3_000
    hotness = rng.random(num_nodes).astype(np.float32) * 0.2
    thr = oracle_mod.flush_thresholds(hotness)
    thr = np.minimum(thr, 3).astype(np.int32)  # short periods so that rows do flush
    cc = ColdCache(f"cc{mode}{dim}", entries, dim, threshold=_t(thr), cnt_threshold=3, num_clients=clients,
                   local_nodes=local_nodes, local_start=1000, lookup_mode=mode)
    ox = oracle_mod.OracleIndex(entries)
    slots = ox.get_capacity()
    ocache = np.zeros((slots, dim), np.float32)
    orem = oracle_mod.OracleStaging(slots, dim, cnt_threshold=3)
    oloc = oracle_mod.OracleStaging(local_nodes, dim, cnt_threshold=3, iter_threshold=thr[1000:1000 + local_nodes])
    for it in range(7):
        # step 0: flush
        gi, gr, gc, gcounts = cc.flush_remote()
        wi, wr, wc, wcounts = orem.flush(ox, clients)
        assert np.array_equal(gcounts.cpu().numpy(), wcounts), it
        assert np.array_equal(gi.cpu().numpy(), wi) and np.array_equal(gc.cpu().numpy(), wc), it
        assert np.array_equal(gr.cpu().numpy(), wr), it
        gi, gr, gc, gcounts = cc.flush_local()
        wi, wr, wc, wcounts = oloc.flush(None, clients)
        assert np.array_equal(gcounts.cpu().numpy(), wcounts), it
        assert np.array_equal(gi.cpu().numpy(), wi) and np.array_equal(gr.cpu().numpy(), wr), it
        assert np.array_equal(gc.cpu().numpy(), wc), it
        # step 2: insert uncached embeddings
        new_ids = rng.integers(0, num_nodes, 900, dtype=np.int64)
        embs = rng.standard_normal((900, dim)).astype(np.float32)
        # duplicate ids inside a batch carry the same row
        uniq_rows = {}
        for k, i in enumerate(new_ids):
            uniq_rows.setdefault(int(i), embs[k])
            embs[k] = uniq_rows[int(i)]
        glocs = cc.insert(_t(new_ids), _t(embs))
        wlocs = orem.insert(ox, new_ids, embs, ocache)
        assert np.array_equal(glocs.cpu().numpy(), wlocs), it
        assert np.array_equal(cc.emb.cpu().numpy(), ocache), it
        # step 3: accumulate, two "clients", unique ids per message
        for c in range(2):
            ids = rng.permutation(num_nodes)[:1500].astype(np.int64)
            g = (rng.standard_normal((1500, dim)) * 1e-3).astype(np.float32)
            cc.accumulate_remote(_t(ids), _t(g))
            orem.accumulate_cached(ox, ids, g, thr, 1)
            lids = (1000 + rng.permutation(local_nodes)[:700]).astype(np.int64)
            lg = (rng.standard_normal((700, dim)) * 1e-3).astype(np.float32)
            cc.accumulate_local(_t(lids), _t(lg))
            oloc.accumulate_direct(lids, lg, 1000, 1)
        for name, gs, os_ in (("remote", cc.remote, orem), ("local", cc.local, oloc)):
            assert np.array_equal(gs.cnt.cpu().numpy(), os_.cnt), (it, name)
            assert np.array_equal(gs.idx.cpu().numpy(), os_.idx), (it, name)
            assert np.array_equal(gs.iter_count.cpu().numpy(), os_.iter_count), (it, name)
            assert np.array_equal(gs.iter_threshold.cpu().numpy(), os_.iter_threshold), (it, name)
            assert np.array_equal(gs.grad.cpu().numpy(), os_.grad), (it, name)
        gi, gl = cc.index.export_state()
        oi, ol = ox.export()
        assert np.array_equal(gi.cpu().numpy(), oi) and np.array_equal(gl.cpu().numpy(), ol), it
    assert int(cc.dropped.item()) > 0


@pytest.mark.parametrize("emb_dtype", [np.float32, np.float16])
@pytest.mark.parametrize("dim", [3, 64, 128])
def test_sparse_adam(cuda_lib, oracle_mod, emb_dtype, dim):
    """Three steps of SparseAdam on an owner shard (id % 4 == 1): state and embedding within
    1e-5 relative of the fp32 restatement (fp16 tables: within one fp16 rounding)."""
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdam

    rng = np.random.default_rng(dim)
    num, world, rank = 40_000, 4, 1
    emb = ShardedEmbedding(num, dim, rank, world, dtype=torch.float16 if emb_dtype == np.float16 else torch.float32)
    w0 = (rng.standard_normal((emb.rows, dim)) * 0.01).astype(emb_dtype)
    emb.weight.copy_(_t(w0))
    opt = SparseAdam(emb, lr=0.01)
    step = np.zeros(emb.rows, np.float32)
    mem = np.zeros((emb.rows, dim), np.float32)
    power = np.zeros((emb.rows, dim), np.float32)
    w = w0.copy()
    for it in range(3):
        local_rows = rng.permutation(emb.rows)[:3000]
        ids = (local_rows * world + rank).astype(np.int64)
        g = (rng.standard_normal((3000, dim)) * 1e-3).astype(np.float32)
        cnt = rng.integers(1, 5, 3000, dtype=np.int64) if it == 1 else None
        opt.update(_t(ids), _t(g), None if cnt is None else _t(cnt), is_unique=True)
        oracle_mod.sparse_adam_update(ids, g, step, mem, power, w, 0.01, cnt=cnt, id_offset=rank, id_stride=world)
        assert np.array_equal(opt.state_step.cpu().numpy(), step)
        # 1e-5 relative to the size of the operands: a sum of two terms of opposite sign can
        # cancel, so the bound is on |a| + |b| (gradients ~1e-3, updates ~lr = 1e-2), not on the result
        np.testing.assert_allclose(opt.state_mem.cpu().numpy(), mem, rtol=RTOL, atol=RTOL * 1e-3)
        np.testing.assert_allclose(opt.state_power.cpu().numpy(), power, rtol=RTOL, atol=RTOL * 1e-6)
        if emb_dtype == np.float32:
            np.testing.assert_allclose(emb.weight.cpu().numpy(), w, rtol=RTOL, atol=RTOL * 2e-2)
        else:
            got = emb.weight.float().cpu().numpy()
            assert np.abs(got - w.astype(np.float32)).max() <= 2e-5  # one fp16 ulp near 0.03
            w = emb.weight.cpu().numpy().copy()  # keep the two tables from drifting apart by roundings


def test_sparse_adam_not_unique_uses_mean(cuda_lib, oracle_mod):
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdam

    rng = np.random.default_rng(1)
    emb = ShardedEmbedding(5000, 32)
    opt = SparseAdam(emb, lr=0.05)
    ids = rng.integers(0, 5000, 20_000, dtype=np.int64)
    g = (rng.standard_normal((20_000, 32)) * 1e-3).astype(np.float32)
    opt.update(_t(ids), _t(g), id_bits=16)
    u, mean, _ = oracle_mod.unique_grads(ids, g)
    step = np.zeros(5000, np.float32)
    mem = np.zeros((5000, 32), np.float32)
    power = np.zeros((5000, 32), np.float32)
    w = np.zeros((5000, 32), np.float32)
    oracle_mod.sparse_adam_update(u, mean, step, mem, power, w, 0.05)
    assert np.array_equal(opt.state_step.cpu().numpy(), step)
    # the first Adam step is lr * g / (|g| + eps): where the duplicates of an id nearly cancel,
    # the rounding of the mean is amplified by 1/|g|, so the bound is relative to lr
    np.testing.assert_allclose(emb.weight.cpu().numpy(), w, rtol=1e-4, atol=0.05 * 1e-3)


@pytest.mark.parametrize("emb_dtype", [np.float32, np.float16])
def test_sparse_adagrad(cuda_lib, oracle_mod, emb_dtype):
    """Configuration-4 shapes scaled down: 64-dim fp32 gradients, fp16 table sharded id % 8."""
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad

    rng = np.random.default_rng(3)
    num, world, rank, dim = 80_000, 8, 5, 64
    emb = ShardedEmbedding(num, dim, rank, world, dtype=torch.float16 if emb_dtype == np.float16 else torch.float32)
    w = (rng.standard_normal((emb.rows, dim)) * 0.01).astype(emb_dtype)
    emb.weight.copy_(_t(w))
    opt = SparseAdagrad(emb, lr=0.01)
    ssum = np.zeros((emb.rows, dim), np.float32)
    for it in range(3):
        rows = rng.permutation(emb.rows)[:4000]
        ids = (rows * world + rank).astype(np.int64)
        g = (rng.standard_normal((4000, dim)) * 1e-3).astype(np.float32)
        opt.update(_t(ids), _t(g), is_unique=True)
        oracle_mod.sparse_adagrad_update(ids, g, ssum, w, 0.01, id_offset=rank, id_stride=world)
        np.testing.assert_allclose(opt.state_sum.cpu().numpy(), ssum, rtol=RTOL, atol=RTOL * 1e-6)
        if emb_dtype == np.float32:
            np.testing.assert_allclose(emb.weight.cpu().numpy(), w, rtol=RTOL, atol=RTOL * 2e-2)
        else:
            got = emb.weight.float().cpu().numpy()
            assert np.abs(got - w.astype(np.float32)).max() <= 2e-5
            w = emb.weight.cpu().numpy().copy()


@pytest.mark.parametrize("unique", [True, False])
def test_sparse_adam_state_through_the_tiered_cache(cuda_lib, unique):
    """Optimiser state in pinned host memory behind LocalSparseAdamStateCache (a third of the
    rows cached in HBM, python/EmbCache/cache.py:66-194 used at sparse_optim.py:621-668) against
    the all-HBM optimiser on the same updates: the same kernel runs on the same numbers, so
    state and weights are bit-exact."""
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdam

    rng = np.random.default_rng(11)
    num, dim, world, rank = 24_000, 32, 2, 1
    ea, eb = ShardedEmbedding(num, dim, rank, world), ShardedEmbedding(num, dim, rank, world)
    w0 = (rng.standard_normal((ea.rows, dim)) * 0.01).astype(np.float32)
    ea.weight.copy_(_t(w0))
    eb.weight.copy_(_t(w0))
    full = ea.rows * (4 + 8 * dim)
    hot = torch.from_numpy(rng.random(ea.rows).astype(np.float32))
    a = SparseAdam(ea, lr=0.01)
    b = SparseAdam(eb, lr=0.01, state_budget_bytes=full // 3, hotness=hot)
    assert a.state_cache is None and b.state_cache is not None and b.state_cache.has_cached
    assert not b.state_mem.is_cuda and b.state_mem.is_pinned()
    cached_rows = int((b.state_cache.idx_map != -1).sum().item())
    assert 0 < cached_rows < ea.rows
    for it in range(4):
        if unique:
            ids = (rng.permutation(ea.rows)[:3000] * world + rank).astype(np.int64)
        else:
            ids = (rng.integers(0, ea.rows, 5000) * world + rank).astype(np.int64)
        g = (rng.standard_normal((ids.size, dim)) * 1e-3).astype(np.float32)
        cnt = rng.integers(1, 5, ids.size, dtype=np.int64) if it % 2 else None
        for opt in (a, b):
            opt.update(_t(ids), _t(g), None if cnt is None else _t(cnt), is_unique=unique, id_bits=20)
        for x, y in zip(a.full_state(), b.full_state()):
            assert torch.equal(x, y), it
        assert torch.equal(ea.weight, eb.weight), it
    # the backing tensors hold the rows that are not cached, the HBM copy the others
    idx_map = b.state_cache.idx_map.cpu()
    uncached = torch.nonzero(idx_map == -1).flatten()
    assert torch.equal(b.state_mem[uncached], a.state_mem.cpu()[uncached])


@pytest.mark.parametrize("slots,dim,cap", [(1, 4, 0), (31, 3, 0), (1023, 128, 0), (1024, 128, 100), (1025, 1, 0),
                                           (40_000, 130, 0), (40_000, 260, 7_000), (4_194_304 + 1_500, 2, 0)])
@pytest.mark.parametrize("share", [0.0, 0.03, 1.0])
@pytest.mark.parametrize("sync", [True, False])
def test_flush_to_one_client(cuda_lib, slots, dim, cap, share, sync):
    """The whole table after a flush and what left, bit for bit, at the edges of the 1,024 slots a block
    takes at a time, with several rounds a block (over 4,194,304 slots), an output smaller than the
    stale rows, none or all slots stale, and rows of vectors and of single floats."""
    from hades_b200.cold_cache import StagingTable

    rng = np.random.default_rng(slots + dim)
    t = StagingTable(slots, dim, "cuda")
    grad = rng.standard_normal((slots, dim)).astype(np.float32)
    cnt = rng.integers(-1, 4, slots).astype(np.int32)
    age = rng.integers(0, 5, slots).astype(np.int32)
    stale = rng.random(slots) < share
    cnt[stale] = np.maximum(cnt[stale], 1)
    limit = np.where(stale, age, age + 1).astype(np.int32)
    often = stale & (rng.random(slots) < 0.3)
    limit[often] += 5
    cnt[often] = 16
    ids = rng.permutation(slots).astype(np.int64)
    ids[rng.random(slots) < 0.01] = -1
    for dst, src in ((t.grad, grad), (t.cnt, cnt), (t.idx, ids), (t.iter_count, age), (t.iter_threshold, limit)):
        dst.copy_(_t(src))
    found = np.nonzero(stale & (ids >= 0))[0]
    left = found[:cap] if cap else found
    got_ids, got_rows, got_cnt, counts = t.flush(None, 16, 1, sync, cap)
    if sync:
        assert t.last_counts_host == [found.size]
    else:
        got_ids, got_rows, got_cnt = got_ids[:left.size], got_rows[:left.size], got_cnt[:left.size]
    assert counts.tolist() == [found.size]
    assert np.array_equal(got_ids.cpu().numpy(), ids[left])
    assert np.array_equal(got_cnt.cpu().numpy(), cnt[left])
    assert np.array_equal(got_rows.cpu().numpy(), grad[left])
    stays = cnt > 0
    stays[left] = False
    age[stays] += 1
    age[left], cnt[left], grad[left] = 0, 0, 0
    for dst, want in ((t.grad, grad), (t.cnt, cnt), (t.idx, ids), (t.iter_count, age), (t.iter_threshold, limit)):
        assert np.array_equal(dst.cpu().numpy(), want)


def test_early_launches_come_behind_events_and_copies(cuda_lib):
    """Kernels whose blocks take their places under the kernel before them still see what the stream waited for in
    between: another stream's writes behind an event, a copy, a kernel that is not this library's."""
    from hades_b200.cold_cache import ColdCache

    dev, n, dim = torch.device("cuda"), 4096, 128
    cold = ColdCache("early_launch", 8 * n, dim)
    ids = torch.arange(n, device=dev)
    cold.insert(ids, torch.zeros((n, dim), device=dev))
    torch.cuda.synchronize()
    host = torch.full((n, dim), 2.0).pin_memory()
    grads, other, main = torch.zeros((n, dim), device=dev), torch.cuda.Stream(), torch.cuda.Stream()
    for rnd in range(3):
        grads.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            torch.cuda._sleep(20_000_000)
            grads.fill_(1.0)
            written = other.record_event()
        with torch.cuda.stream(main):
            cold.accumulate_remote(ids, grads * 0)
            main.wait_event(written)
            cold.accumulate_remote(ids, grads)        # 1
            torch.cuda._sleep(5_000_000)
            grads.copy_(host, non_blocking=True)
            cold.accumulate_remote(ids, grads)        # 2
            grads.mul_(2.0)
            cold.accumulate_remote(ids, grads)        # 4
        torch.cuda.synchronize()
        slots = cold.index.cuda_lookup_found(ids)[0]
        assert torch.equal(cold.remote.grad[slots], torch.full((n, dim), 7.0 * (rnd + 1), device=dev)), rnd


@pytest.mark.parametrize("emb_dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("kind", ["adam", "adagrad"])
@pytest.mark.parametrize("n,dim", [(1, 8), (33, 24), (257, 16), (1000, 128), (700, 256), (90, 264), (40, 1032)])
def test_updates_of_8_values_a_lane_have_the_bits_of_4(cuda_lib, emb_dtype, kind, n, dim):
    """Rows of a multiple of 8 columns move 32 bytes a lane where their buffers begin at 32 bytes; gradients that
    begin 16 bytes further take the form of 16 bytes a lane.  The values are worked out alike: the same bits."""
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad, SparseAdam

    g = torch.Generator(device="cuda")
    g.manual_seed(n * dim)
    results = []
    w0 = torch.randn((2 * n + 5, dim), device="cuda", generator=g) * 0.01
    ids = torch.randperm(2 * n + 5, device="cuda", generator=g)[:n]
    flat = torch.randn(n * dim + 4, device="cuda", generator=g) * 1e-3
    cnt = torch.randint(1, 5, (n,), device="cuda", generator=g)
    for offset in (0, 4):
        grads = torch.empty(n * dim + 8, device="cuda")[offset:offset + n * dim].view(n, dim)
        grads.copy_(flat[:n * dim].view(n, dim))
        assert grads.data_ptr() % 32 == 4 * offset
        emb = ShardedEmbedding(2 * n + 5, dim, dtype=emb_dtype)
        emb.weight.copy_(w0)
        opt = (SparseAdam if kind == "adam" else SparseAdagrad)(emb, lr=0.01)
        for c in (None, cnt):
            opt.update(ids, grads, c, is_unique=True)
        results.append([emb.weight.clone()] + [v.clone() for v in vars(opt).values() if isinstance(v, torch.Tensor)])
    assert not torch.equal(results[0][0].float(), w0)
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("emb_dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("kind,n,dim", [("adam", 56_833, 8), ("adagrad", 60_001, 8), ("adam", 28_417, 16), ("adagrad", 14_209, 24),
                                        ("adam", 14_209, 32), ("adam", 33, 40), ("adagrad", 2_369, 256), ("adagrad", 1_149, 528)])
def test_larger_updates_of_8_values_a_lane_have_the_bits_of_4(cuda_lib, emb_dtype, kind, n, dim):
    test_updates_of_8_values_a_lane_have_the_bits_of_4(cuda_lib, emb_dtype, kind, n, dim)


@pytest.mark.parametrize("kind,n,dim,values", [
    ("adam", 2_000, 32, 4), ("adagrad", 2_000, 8, 4), ("adam", 56_832, 8, 4), ("adam", 56_833, 8, 8), ("adagrad", 28_416, 16, 4),
    ("adagrad", 28_417, 16, 8), ("adam", 14_208, 24, 4), ("adam", 14_209, 32, 8), ("adam", 100, 40, 8), ("adagrad", 100, 64, 8),
    ("adam", 100, 256, 8), ("adagrad", 2_368, 256, 4), ("adagrad", 2_369, 256, 8), ("adagrad", 100, 248, 8), ("adam", 60_000, 100, 4)])
def test_values_a_lane_of_updates(cuda_lib, kernels_of, kind, n, dim, values):
    """Narrow rows move 32 bytes a lane where the warps of 16 bytes a lane would not all run at once."""
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad, SparseAdam

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are those of 148 SMs")
    opt = (SparseAdam if kind == "adam" else SparseAdagrad)(ShardedEmbedding(n, dim), lr=0.01)
    ids, grads = torch.arange(n, device="cuda"), torch.zeros((n, dim), device="cuda")
    k, = [k for k in kernels_of(lambda: opt.update(ids, grads, None, is_unique=True)) if "sparse_update" in k["name"]]
    assert k["arguments"][-1] == values, k
