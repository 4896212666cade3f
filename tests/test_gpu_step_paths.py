"""The one-trainer step as two library calls (``hb_step_forward`` / ``hb_step_backward``) against the same step
composed of separate operators, and what it has to follow, refuse or leave to the composed form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _small(name, dim=32, batch=4096, flush_every=3):
    from hades_b200 import synth

    return synth.CacheFetchConfig(name, 1, 30_000, dim, 3000, batch, 1.1, flush_every=flush_every)


def _steps(cfg, n, seed=3):
    from hades_b200 import synth

    rng = synth.rng_for(1, 0, seed)
    sampler = synth.ZipfSampler(cfg.table_rows, cfg.zipf_s)
    return [(torch.from_numpy(sampler.ids(rng, cfg.batch)).cuda(),
             torch.from_numpy(synth.normal_rows(rng, cfg.batch, cfg.dim, cfg.grad_sigma)).cuda()) for _ in range(n)]


def _state(path):
    r = path.cold.remote
    out = {"table": path.table, "cache": path.cold.emb, "staged": r.grad, "cnt": r.cnt, "iter": r.iter_count,
           "thr": r.iter_threshold, "dropped": path.cold.dropped}
    out.update({k: v for k, v in vars(path.opt).items() if isinstance(v, torch.Tensor)})
    out["line_ids"], out["lru"] = path.cold.index.export_state()
    return out


def _pair(name, **kw):
    """The step as two library calls, and composed of separate operators."""
    from hades_b200 import pipeline

    dim = kw.pop("dim", 32)
    a = pipeline.build_path(_small(name + "_a", dim), **kw)
    b = pipeline.build_path(_small(name + "_b", dim), **kw)
    assert a._one is not None
    b._one = None
    return a, b


def _run_pair(a, b, batches):
    for ids, g in batches:
        ra, rb = a.step(ids, g), b.step(ids, g)
        assert torch.equal(ra[0], rb[0]) and torch.equal(ra[2], rb[2])
    sa, sb = _state(a), _state(b)
    for k in sb:
        assert torch.equal(sa[k], sb[k]), k


def test_table_of_an_unsupported_type_is_refused(cuda_lib):
    from hades_b200 import pipeline

    cfg = _small("fp64_shard")
    path = pipeline.build_path(cfg, table_dtype=torch.float64)
    weight = path.opt.emb.weight.clone()
    (ids, g), = _steps(cfg, 1)
    with pytest.raises(RuntimeError, match=r"fp32 \(4\) or fp16 \(2\)"):
        path.step(ids, g)
    assert torch.equal(path.opt.emb.weight, weight)


@pytest.mark.parametrize("what", ["adagrad", "fresh_adam", "eps", "threshold", "dropped", "staging", "class_table"])
def test_attributes_of_the_path_may_change_between_steps(cuda_lib, what):
    from hades_b200.cold_cache import StagingTable
    from hades_b200.sparse_optim import SparseAdagrad, SparseAdam

    a, b = _pair("attr_" + what)
    batches = _steps(_small("attr"), 8)
    _run_pair(a, b, batches[:4])
    old = []  # what was in use stays allocated
    for p in (a, b):
        old.append(dict(vars(p)))
        if what == "adagrad":
            p.opt = SparseAdagrad(p.opt.emb, lr=0.01)
        elif what == "fresh_adam":
            old.append(p.opt)
            p.opt = SparseAdam(p.opt.emb, lr=0.01)
        elif what == "eps":
            p.opt._eps = 1e-2
        elif what == "threshold":
            old.append(p.cold.threshold)
            p.cold.threshold = torch.full((p.num_nodes,), 2, dtype=torch.int32, device="cuda")
        elif what == "dropped":
            old.append(p.cold.dropped)
            p.cold.dropped = torch.zeros(1, dtype=torch.int64, device="cuda")
        elif what == "staging":
            old.append(p.cold.remote)
            p.cold.remote = StagingTable(p.cold.remote.slots, p.dim, p.cold.emb.device)
        elif what == "class_table":
            p.class_table = torch.full_like(p.class_table, 2)
    _run_pair(a, b, batches[4:])


def test_optimizer_of_the_users_own_is_called(cuda_lib):
    from hades_b200.sparse_optim import SparseAdam

    class Clipped(SparseAdam):
        calls = 0

        def update(self, idx, grad, *args, **kw):
            Clipped.calls += 1
            return super().update(idx, grad.clamp(-1e-4, 1e-4), *args, **kw)

    from hades_b200 import pipeline

    cfg = _small("own_opt")
    p = pipeline.build_path(cfg)
    q = pipeline.EmbeddingPath(p.table, p.class_table, p.cold, Clipped(p.opt.emb, lr=0.01), flush_every=3, id_bits=p.id_bits)
    (ids, g), = _steps(cfg, 1)
    q.step(ids, g)
    assert Clipped.calls == 1


@pytest.mark.parametrize("what,why", [("wide_classes", "int8"), ("host_table", "pinned host memory"),
                                      ("strided_table", "contiguous"), ("narrow_table", r"size\(1\)")])
def test_tensors_that_do_not_fit_are_refused(cuda_lib, what, why):
    from hades_b200 import pipeline

    cfg = _small("misfit_" + what)
    path = pipeline.build_path(cfg)
    (ids, g), = _steps(cfg, 1)
    if what == "wide_classes":
        path.class_table = path.class_table.long()
    elif what == "host_table":
        path.table = path.table.cpu()
    elif what == "strided_table":
        path.table = torch.cat([path.table, path.table], 1)[:, :cfg.dim]
    else:
        path.table = path.table[:, : cfg.dim // 2].contiguous()
    before = _state(path)
    with pytest.raises(RuntimeError, match=why):
        path.forward(ids)
    after = _state(path)
    assert all(torch.equal(before[k], after[k]) for k in before)


def test_sorted_view_stays_fresh_where_nothing_is_inserted(cuda_lib):
    from hades_b200 import EmbCacheLib as E
    from hades_b200 import pipeline

    cfg = _small("sorted_noinsert", flush_every=0)
    paths = [pipeline.build_path(_small(f"sorted_noinsert_{k}", flush_every=0), lookup_mode=E.LOOKUP_SORTED, insert_misses=False)
             for k in range(2)]
    batches = _steps(cfg, 6)
    outs = [torch.empty((cfg.batch, cfg.dim), device="cuda") for _ in paths]
    for ids, _ in batches[:2]:
        for p, o in zip(paths, outs):
            p.step(ids, batches[0][1], o)
    buf = torch.empty_like(batches[0][0])
    paths[1].capture(buf, batches[0][1], outs[1])
    for ids, _ in batches[2:]:
        r = [p.step(ids, batches[0][1], o) for p, o in zip(paths, outs)]
        assert torch.equal(r[0][0], r[1][0]) and torch.equal(r[0][2], r[1][2])
    sa, sb = _state(paths[0]), _state(paths[1])
    for k in sa:
        assert torch.equal(sa[k], sb[k]), k


def test_sorted_view_follows_insertions(cuda_lib):
    from hades_b200 import EmbCacheLib as E

    _run_pair(*_pair("sorted_insert", lookup_mode=E.LOOKUP_SORTED), _steps(_small("sorted_insert"), 7))


@pytest.mark.parametrize("optimizer", ["adam", "adagrad"])
@pytest.mark.parametrize("dim", [3, 47, 127])
def test_rows_of_odd_width_as_composed(cuda_lib, dim, optimizer):
    """Columns one by one: counts and bias corrections divide in both forms."""
    a, b = _pair(f"odd_{dim}_{optimizer}", dim=dim, optimizer=optimizer)
    _run_pair(a, b, _steps(_small("odd", dim), 7))


@pytest.mark.parametrize("flags", [{}, {"insert_misses": False}, {"touch_lru": False},
                                   {"insert_misses": False, "touch_lru": False}], ids=lambda f: "_".join(f) or "default")
@pytest.mark.parametrize("n", [1, 33, 513, 8191, 8192, 8193])
def test_runs_looked_up_in_the_launch_of_the_sort(cuda_lib, n, flags):
    """Up to 8,192 ids a run is looked up where the sort writes it, above in a launch of its own; the runs of a warp
    lie in two chunks of 32, whose counts cut the list of misses (miss_cap)."""
    a, b = _pair(f"resolve_{n}_" + "_".join(flags), **flags)
    a.miss_cap = b.miss_cap = max(n // 8, 1)
    _run_pair(a, b, [(ids[:n], g[:n]) for ids, g in _steps(_small("resolve", batch=8193), 4, seed=n)])


@pytest.mark.parametrize("n", [40, 8192, 8193])
def test_ids_outside_of_the_table_as_composed(cuda_lib, n):
    """Negative ids are a run of their own, which sorts last; ids behind the table have no class and no row.  Their
    output rows stay as they were, the status word tells."""
    from hades_b200 import _lib

    a, b = _pair(f"outside_{n}")
    for ids, g in _steps(_small("outside", batch=n), 3, seed=n):
        ids[::7], ids[3::11] = -1, 30_000 + n % 2000
        outs = [torch.full_like(g, 7.0) for _ in range(2)]
        ra, rb = a.step(ids, g, outs[0]), b.step(ids, g, outs[1])
        assert _lib.device_status() != 0
        assert torch.equal(outs[0], outs[1]) and torch.equal(ra[2], rb[2])
        assert (outs[0][ids < 0] == 7.0).all() and (outs[0][ids >= 30_000] == 7.0).all()
    sa, sb = _state(a), _state(b)
    for k in sb:
        assert torch.equal(sa[k], sb[k]), k


@pytest.mark.parametrize("n,aside,optimizer,mode,miss_cap,dim", [
    (100_000, False, "adam", 0, 1 << 17, 32), (100_000, True, "adagrad", 0, 700, 32),
    (100_001, False, "adam", 0, 700, 32), (100_001, True, "adam", 0, 1 << 17, 32), (100_001, True, "adagrad", 1, 700, 32),
    (150_001, False, "adagrad", 1, 1 << 17, 3), (150_001, True, "adam", 0, 700, 47), (282_624, True, "adam", 1, 1 << 17, 16),
    (303_105, False, "adam", 0, 1 << 17, 128)])
def test_steps_with_a_second_pass_as_composed(cuda_lib, n, aside, optimizer, mode, miss_cap, dim):
    """Above 70,000 ids sums, the lookup of the cold ids on the second stream and the update with the ageing in it;
    with and without a fetch aside, through step() and through its two halves, over several flushes, and with
    gradients of another batch than the last one fetched."""
    a, b = _pair(f"second_{n}_{aside}_{optimizer}_{mode}", dim=dim, optimizer=optimizer, lookup_mode=mode)
    for p in (a, b):
        p.overlap_fetch, p.miss_cap = aside, miss_cap
    batches = _steps(_small("second", dim, batch=n), 5)
    for k, (ids, g) in enumerate(batches):
        rows = []
        for p in (a, b):
            if k % 2 == 0:
                rows.append(p.step(ids, g))
            else:
                rows.append(p.forward(ids, join=False, on_side=aside))
                p.backward(*((ids, g) if k == 1 else batches[0]))
                if k == 3:
                    torch.cuda.synchronize()
        assert torch.equal(rows[0][0], rows[1][0]) and torch.equal(rows[0][2], rows[1][2]), k
    sa, sb = _state(a), _state(b)
    for k in sb:
        assert torch.equal(sa[k], sb[k]), k


@pytest.mark.parametrize("optimizer", ["adam", "adagrad"])
@pytest.mark.parametrize("dim", [3, 16, 47, 100, 127, 128, 256, 512])
def test_steps_at_the_line_of_updates_at_once(cuda_lib, optimizer, dim):
    """70,000 ids are updated as their sums become complete, one more in a launch of its own: the state is that of the
    composed step, and the launches say which it was."""
    launches = []
    for n in (70_000, 70_001):
        a, b = _pair(f"line_{n}_{optimizer}_{dim}", dim=dim, optimizer=optimizer)
        batches = _steps(_small("line", dim, batch=n), 3)
        _run_pair(a, b, batches)
        a.forward(batches[0][0], join=False)
        before = cuda_lib.hb_launch_count()
        a.backward(*batches[0])
        launches.append(cuda_lib.hb_launch_count() - before)
    assert launches[1] == launches[0] + 1


@pytest.mark.parametrize("optimizer,dim", [("adam", 47), ("adam", 127), ("adam", 128), ("adam", 256), ("adagrad", 47),
                                           ("adagrad", 127), ("adagrad", 256), ("adagrad", 320)])
def test_the_second_pass_has_the_blocks_that_run_at_once(cuda_lib, kernels_of, optimizer, dim):
    """As many as the registers of its form leave room for, whatever its rows, and one per 256 ids below that."""
    n = 160_001
    a, _ = _pair(f"blocks_{optimizer}_{dim}", dim=dim, optimizer=optimizer, touch_lru=False)
    (ids, g), = _steps(_small("blocks", dim, batch=n), 1)
    second = [k for k in kernels_of(lambda: a.step(ids, g)) if "step_apply_kernel" in k["name"]]
    assert len(second) == 1
    for k in second:
        warps = 65_536 // (32 * (-(-k["registers"] // 8) * 8))
        fit = warps // (k["block"] // 32) * torch.cuda.get_device_properties(0).multi_processor_count
        assert k["grid"] == min(fit, -(-n // 256)), k


@pytest.mark.parametrize("optimizer", ["adam", "adagrad"])
def test_backward_comes_behind_the_callers_stream(cuda_lib, optimizer):
    """What the caller enqueues between a fetch aside and its backward pass is seen by the lookup of the cold ids, which
    runs on the step's second stream in steps of more than 70,000 ids."""
    n = 100_001
    a, b = _pair("behind_" + optimizer, optimizer=optimizer)
    for p in (a, b):
        p.cold.threshold = torch.full((p.num_nodes,), 1, dtype=torch.int32, device="cuda")
        p.miss_cap = 500  # the cold ids beyond it are dropped
    for rnd, (ids, g) in enumerate(_steps(_small("behind", batch=n), 4)):
        rows = []
        for p, aside in ((a, True), (b, False)):
            rows.append(p.forward(ids, on_side=aside))
            torch.cuda._sleep(20_000_000)
            p.cold.threshold.fill_(rnd + 2)
            p.cold.dropped.zero_()
            p.backward(ids, g)
        assert torch.equal(rows[0][0], rows[1][0]) and torch.equal(rows[0][2], rows[1][2])
        assert a.cold.dropped.item() > 0
        sa, sb = _state(a), _state(b)
        for k in sb:
            assert torch.equal(sa[k], sb[k]), (rnd, k)


def test_capture_behind_a_fetch_aside_is_refused(cuda_lib):
    """A fetch enqueued outside of a capture cannot be waited for inside it; nothing of the call runs."""
    import ctypes

    cu, n = ctypes.CDLL("libcuda.so.1"), 100_001
    a, b = _pair("aside_capture")
    (ids, g), (ids2, g2) = _steps(_small("aside_capture", batch=n), 2)
    other = torch.cuda.Stream()
    a.forward(ids, on_side=True)
    b.forward(ids)
    torch.cuda.synchronize()
    before = _state(a)
    graph = ctypes.c_void_p()
    with torch.cuda.stream(other):
        assert cu.cuStreamBeginCapture_v2(ctypes.c_void_p(other.cuda_stream), 1) == 0
        with pytest.raises(RuntimeError):
            a._backward_core(ids, g)
        assert cu.cuStreamEndCapture(ctypes.c_void_p(other.cuda_stream), ctypes.byref(graph)) != 0
    ctypes.CDLL("libcudart.so.12").cudaGetLastError()
    torch.cuda.synchronize()
    after = _state(a)
    assert all(torch.equal(before[k], after[k]) for k in before)
    a.backward(ids, g)
    b.backward(ids, g)
    _run_pair(a, b, [(ids2, g2)])


def test_other_streams_run_beside_the_sort(cuda_lib):
    """The launch behind the sort does not wait in the places of kernels of other streams.  Three small ones take a
    twelfth of the step's time beside it; behind its sort they would take two fifths."""
    from hades_b200 import pipeline, synth

    cfg = synth.CacheFetchConfig("beside", 1, 300_000, 128, 30_000, 280_000, 1.1, flush_every=0)
    path = pipeline.build_path(cfg)
    (ids, g), = _steps(cfg, 1)
    out, small = torch.empty_like(g), torch.ones(1 << 16, device="cuda")
    gate, main, other = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    beside, step = [], []
    for rnd in range(40):
        at = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        with torch.cuda.stream(gate):
            torch.cuda._sleep(1_000_000)
            opened = gate.record_event()
        with torch.cuda.stream(main):
            main.wait_event(opened)
            at[0].record()
            path.step(ids, g, out)
            at[1].record()
        with torch.cuda.stream(other):
            other.wait_event(opened)
            at[2].record()
            for _ in range(3):
                small.add_(1)
            at[3].record()
        torch.cuda.synchronize()
        step.append(at[0].elapsed_time(at[1]))
        beside.append(at[2].elapsed_time(at[3]))
    assert sorted(beside)[20] < 0.2 * sorted(step)[20], (sorted(beside)[20], sorted(step)[20])


@pytest.mark.parametrize("dim", [16, 100, 128, 256, 512])
@pytest.mark.parametrize("n,length", [(1, 1), (63, 1), (64, 64), (65, 7), (130, 129), (1000, 1000), (5000, 37), (5000, 1),
                                      (40_000, 3), (40_000, 900)])
def test_runs_of_every_length_updated_by_the_ctas_that_sum_them(cuda_lib, n, length, dim):
    """Runs inside a piece, across pieces, across CTAs and across many of them, and batches that end inside a CTA's
    share: the same bits as sums and update one after the other."""
    a, b = _pair(f"runs_{n}_{length}_{dim}", dim=dim, optimizer="adam")
    g = torch.Generator(device="cuda")
    g.manual_seed(n + length + dim)
    batches = []
    for _ in range(2):
        distinct = torch.randperm(30_000, device="cuda", generator=g)[:max(min(n // length, 30_000), 1)]
        ids = distinct[torch.arange(n, device="cuda") % distinct.numel()]
        batches.append((ids[torch.randperm(n, device="cuda", generator=g)], torch.randn((n, dim), device="cuda", generator=g) * 1e-3))
    _run_pair(a, b, batches)
