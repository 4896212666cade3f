"""Aggregation with the optimiser's update as its output (hb_unique_update_f32, what
``SparseAdam.update`` / ``SparseAdagrad.update`` run on ids that repeat) against a float64
restatement of unique_grads + the update rule (python/EmbCache/sparse_optim.py:142-157,590-685), at
the edges of pieces, CTAs and column layouts."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LR, B1, B2 = 0.01, 0.9, 0.999


def _reference(kind, ids, grads, cnt, w, s0, s1, step, rank, world):
    u, inv = torch.unique(ids, return_inverse=True)
    sums = torch.zeros((u.numel(), grads.size(1)), dtype=torch.float64, device="cuda").index_add_(0, inv, grads.double())
    div = torch.zeros(u.numel(), dtype=torch.float64, device="cuda").index_add_(
        0, inv, torch.ones_like(inv, dtype=torch.float64) if cnt is None else cnt.double())
    g = sums / (div if cnt is None else div + 1)[:, None]
    r = (u - rank) // world
    if kind == "adam":
        step[r] += 1
        s0[r] = B1 * s0[r] + (1 - B1) * g
        s1[r] = B2 * s1[r] + (1 - B2) * g * g
        m, v = s0[r] / (1 - B1 ** step[r])[:, None], s1[r] / (1 - B2 ** step[r])[:, None]
        w[r] -= LR * m / (v.sqrt() + 1e-8)
    else:
        s0[r] += g * g
        w[r] -= LR * g / (s0[r].sqrt() + 1e-10)
    return r


@pytest.mark.parametrize("kind,dtype", [("adam", torch.float32), ("adam", torch.float16), ("adagrad", torch.float32),
                                        ("adagrad", torch.float16)])
@pytest.mark.parametrize("n,dim", [(1, 128), (7, 4), (8, 16), (129, 32), (257, 128), (2049, 47), (4097, 100), (6000, 3),
                                   (70_001, 64), (9_001, 256), (3_001, 512), (40_000, 128), (3_000, 520)])
def test_update_of_repeated_ids(cuda_lib, kind, dtype, n, dim):
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad, SparseAdam

    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + dim)
    rank, world, num = 1, 3, 30_000
    emb = ShardedEmbedding(num, dim, rank, world, dtype=dtype, init_sigma=0.01, seed=n)
    opt = (SparseAdam if kind == "adam" else SparseAdagrad)(emb, lr=LR)
    w = emb.weight.double()
    s0, s1 = torch.zeros_like(w), torch.zeros_like(w)
    step = torch.zeros(emb.rows, dtype=torch.float64, device="cuda")
    for it in range(3):
        # one id with a third of the rows (it crosses CTAs), one with a few, the rest nearly distinct
        rows = torch.randint(0, emb.rows, (n,), device="cuda", generator=gen)
        rows[torch.rand(n, device="cuda", generator=gen) < 0.33] = 17
        rows[:12] = 18
        ids = rows * world + rank
        # values whose sums do not nearly cancel: the first updates of a row are lr * g / |g|
        grads = (1 + torch.rand((n, dim), device="cuda", generator=gen)) * 1e-3
        cnt = torch.randint(1, 5, (n,), device="cuda", generator=gen) if it == 1 else None
        opt.update(ids, grads, cnt, **({"id_bits": 20} if it else {}))
        touched = _reference(kind, ids, grads, cnt, w, s0, s1, step, rank, world)
        if dtype == torch.float16:
            w[touched] = w[touched].half().double()  # the table is rounded after every update
        # Bounds.  State: fp32 sums of n rows and a few roundings, 1e-5.  Adagrad update: the same, of
        # LR: 1e-7, or 1e-4 of the floor 1e-3 below.  Adam update: 1 - beta2^t is at least 1e-3 and comes
        # from fp32 values near 1: 3e-8 (beta2 as fp32) + 1.2e-7 (powf, two units) over 1e-3 is 1.5e-4 of
        # it, 7.5e-5 of its root: with the above under 1e-4 of LR = 1e-6, or 1e-3 of the floor.  fp16
        # table: one unit in the last place (2^-10 of the value) where the exact value lies between two.
        tol = 1e-5
        state0 = opt.state_mem if kind == "adam" else opt.state_sum
        assert float((state0.double() - s0).abs().max() / s0.abs().max()) < tol
        err = (emb.weight.double() - w).abs() / w.abs().clamp(min=1e-3)
        assert float(err.max()) < (2e-3 if dtype == torch.float16 else 1e-3 if kind == "adam" else 1e-4), float(err.max())
        if kind == "adam":
            assert torch.equal(opt.state_step.double(), step)
            assert float((opt.state_power.double() - s1).abs().max() / s1.abs().max()) < tol
        w = emb.weight.double()  # from here on the same table


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("n,dim", [(32_768, 64), (32_769, 3), (32_769, 64), (33_001, 8), (33_001, 16), (33_001, 47),
                                   (33_001, 130), (33_001, 256), (33_001, 512), (33_001, 520)])
def test_adagrad_at_the_edge_of_updating_at_once(cuda_lib, dtype, n, dim):
    """A third of the ids are one id, whose run crosses many CTAs; rows of one pass of the sums, and wider."""
    test_update_of_repeated_ids(cuda_lib, "adagrad", dtype, n, dim)


def _update_in(opt, ids, grads, cnt, id_bits, workspace_bytes):
    """hb_unique_update_f32 with a workspace of that size; its return code."""
    import ctypes as C

    from hades_b200 import _lib

    ws = torch.empty(workspace_bytes, dtype=torch.uint8, device="cuda")
    desc = _lib.OptimDesc(*opt._fields())
    rc = _lib.load().hb_unique_update_f32(ids.data_ptr(), grads.data_ptr(), _lib.ptr(cnt), ids.numel(), None, None, 0,
                                          grads.size(1), id_bits, 1, C.addressof(desc), ws.data_ptr(), workspace_bytes,
                                          _lib.stream_ptr())
    torch.cuda.synchronize()
    return rc


def _workspace_bytes(opt, n, dim, grads):
    import ctypes as C

    from hades_b200 import _lib

    desc = _lib.OptimDesc(*opt._fields())
    return _lib.load().hb_unique_update_workspace_bytes(n, dim, grads.data_ptr(), C.addressof(desc))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("largest,n,dim", [(1_048_576, 437_500, 64), (437_501, 437_500, 64), (2_000_000, 32_768, 16),
                                           (300_000, 4_097, 100), (700_000, 33_001, 47), (300_000, 129, 130),
                                           (200_000, 9_001, 256), (100_000, 33_001, 512), (4_000_000, 1, 8)])
def test_adagrad_in_the_workspace_of_a_larger_batch(cuda_lib, dtype, largest, n, dim):
    """A buffer for the largest batch, which is updated at once, serves smaller ones; one byte below what both need is
    refused and nothing happens."""
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad

    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + dim)
    rank, world, num = 1, 3, 30_000
    emb = ShardedEmbedding(num, dim, rank, world, dtype=dtype, init_sigma=0.01, seed=n)
    opt = SparseAdagrad(emb, lr=LR)
    ids = torch.randint(0, emb.rows, (n,), device="cuda", generator=gen) * world + rank
    grads = (1 + torch.rand((n, dim), device="cuda", generator=gen)) * 1e-3
    cnt = torch.randint(1, 5, (n,), device="cuda", generator=gen)
    given = _workspace_bytes(opt, largest, dim, grads)
    for weights in (None, cnt):
        w, s0 = emb.weight.double(), opt.state_sum.double()
        assert _update_in(opt, ids, grads, weights, 20, given) == 0
        _reference("adagrad", ids, grads, weights, w, s0, None, None, rank, world)
        # (the bounds of test_update_of_repeated_ids)
        assert float((opt.state_sum.double() - s0).abs().max() / s0.abs().max()) < 1e-5
        err = (emb.weight.double() - w).abs() / w.abs().clamp(min=1e-3)
        assert float(err.max()) < (2e-3 if dtype == torch.float16 else 1e-4), float(err.max())
    least = _workspace_bytes(opt, n, dim, grads) - (n * dim * 4 + 255) // 256 * 256
    before = emb.weight.clone()
    assert _update_in(opt, ids, grads, cnt, 20, least - 1) != 0
    assert torch.equal(emb.weight, before)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("n,dim", [(437_500, 64), (437_501, 64), (218_750, 128), (218_751, 128), (224_001, 125),
                                   (54_687, 512), (54_688, 512), (110_001, 256), (280_001, 100), (3_500_001, 8), (600_001, 47)])
def test_adagrad_where_sums_no_longer_fit_in_l2(cuda_lib, dtype, n, dim):
    """Both sides of 28,000,000 values: up to there through memory, beyond it the row is updated when its sum is complete."""
    test_update_of_repeated_ids(cuda_lib, "adagrad", dtype, n, dim)


@pytest.mark.parametrize("kind", ["adam", "adagrad"])
def test_fewer_rows_than_ids_are_refused(cuda_lib, kind):
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad, SparseAdam

    emb = ShardedEmbedding(100, 8, init_sigma=0.01)
    opt = (SparseAdam if kind == "adam" else SparseAdagrad)(emb, lr=LR)
    before = emb.weight.clone()
    with pytest.raises(RuntimeError, match="Check failed"):
        opt.update(torch.arange(20, device="cuda"), torch.ones((19, 8), device="cuda"))
    assert torch.equal(emb.weight, before)


@pytest.mark.parametrize("kind", ["adam", "adagrad"])
@pytest.mark.parametrize("senders,cap,merged", [(1, 40, True), (4, 700, True), (4, 1 << 17, True), (4, (1 << 17) + 1, False),
                                                (5, 700, False)])
def test_ascending_slabs_of_few_senders_are_merged(cuda_lib, monkeypatch, kind, senders, cap, merged):
    """Merged or sorted, the update is that of the slabs as an unsorted list; slabs are empty, part full and full."""
    from hades_b200 import sparse_optim
    from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad, SparseAdam

    calls = []
    merge = sparse_optim._merge_duplicates
    monkeypatch.setattr(sparse_optim, "_merge_duplicates", lambda *a: (calls.append(1), merge(*a))[1])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cap)
    dim, rows = 12, 2 * cap
    opts = []
    for _ in range(2):
        emb = ShardedEmbedding(rows * senders, dim, 0, senders, init_sigma=0.01, seed=3)
        opts.append((SparseAdam if kind == "adam" else SparseAdagrad)(emb, lr=LR))
    ids = torch.zeros((senders, cap), dtype=torch.int64, device="cuda")
    seg = torch.tensor([[cap, 0, cap // 3, 1, cap // 2][s] for s in range(senders)], device="cuda")
    for s in range(senders):
        ids[s] = (torch.randperm(rows, device="cuda", generator=gen)[:cap] * senders).sort().values
    # values whose sums do not nearly cancel: the first updates of a row are lr * g / |g|
    grads = (1 + torch.rand((senders * cap, dim), device="cuda", generator=gen)) * 1e-3
    cnt = torch.randint(1, 5, (senders * cap,), device="cuda", generator=gen)
    for opt, in_order in zip(opts, (True, False)):
        opt.update(ids.flatten(), grads, cnt, seg_counts=seg, seg_cap=cap, sorted_segments=in_order, id_bits=32)
    assert len(calls) == merged
    # sums of up to five rows in another order: a unit or two of fp32
    a, b = (o.emb.weight for o in opts)
    assert float((a - b).abs().max()) < 1e-6 * LR + 2.0**-22 * float(b.abs().max())
