"""The work whose speed counts in this repository: its public calls, over the sizes, types and options they are used
with.

Six kinds of work:

* ``step``       a training step: fetch of a batch's embedding rows through the cache (forward), aggregation of the
                 gradients, owner update of the hot rows, staging of the cold ones, the flush every 8 steps (backward);
                 through ``DistEmb`` and ``DistembSparseGradOptimizer``, or through ``EmbeddingPath.step`` replayed
                 from CUDA graphs
* ``fetch``      lookup and cached fetch without training (evaluation, serving): ``cudaLookupFetch``
* ``aggregate``  sorted unique ids, sums of the duplicates' gradients and counts: ``only_unique_grads``
* ``update``     what an owner does with the rows that its trainers sent: merge of the duplicates and a sparse Adam or
                 Adagrad update, from one unsorted list or from one sorted slab per sender
* ``cold``       one round of the cold-gradient cache: insert, accumulate, flush, update of what left
* ``index``      the id -> slot index called with ids in host memory: lookup with its LRU ageing, add

Ids follow a bounded power law over a popularity ranking that ``synth.rank_to_id`` scatters over the id space, or are
the frontier of a sampled R-MAT graph.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from hades_b200 import EmbCacheLib as E
from hades_b200 import pipeline, synth
from hades_b200.cold_cache import ColdCache, flush_thresholds
from hades_b200.dist_emb import DistEmb, DistembSparseGradOptimizer
from hades_b200.sparse_optim import ShardedEmbedding, SparseAdagrad, SparseAdam, only_unique_grads

DIMS = (16, 32, 64, 100, 128, 256)
TYPES = {"fp32": torch.float32, "fp16": torch.float16, "fp64": torch.float64}
FLUSH_EVERY = 8    # the flush period of the repository's configurations
SENDERS = 8        # trainers of one box that send gradients to an owner
WARM_STEPS = 7     # a measured run begins with the step that flushes


def listed():
    return [
        # a small model in training: what launches and the host cost on each step
        {"name": "step_small", "kind": "step", "nodes": 200_000, "cache": 20_000, "batch": 2_000, "dim": 64, "zipf": 1.1,
         "optimizer": "adagrad", "graph": False, "ids": "gpu"},
        # the batch, table and cache of the repository's first configuration, as a training step
        {"name": "step_65k", "kind": "step", "nodes": 1_000_000, "cache": 100_000, "batch": 65_536, "dim": 128,
         "zipf": 1.1, "optimizer": "adam", "graph": False, "ids": "gpu"},
        # 2-layer GraphSAGE, 1,024 seeds, fanout [25, 10]: frontiers of differing length from a sampler on the host
        {"name": "step_graphsage", "kind": "step", "rmat_bits": 24, "seeds": 1_024, "batch": 282_624, "dim": 128,
         "optimizer": "adam", "graph": False, "ids": "host"},
        # the repository's benchmark: 20 M rows, 4 M cached, 2 M ids per step, replayed from CUDA graphs
        {"name": "step_2m", "kind": "step", "nodes": 20_000_000, "cache": 4_000_000, "batch": 2_000_000, "dim": 128,
         "zipf": 1.2, "optimizer": "adam", "graph": True, "ids": "gpu"},
        # one request of a server, rows of the width of a products feature
        {"name": "fetch_1k", "kind": "fetch", "nodes": 1_000_000, "cache": 100_000, "batch": 1_000, "dim": 100,
         "zipf": 1.1, "type": "fp32"},
        # evaluation over a large batch
        {"name": "fetch_2m", "kind": "fetch", "nodes": 20_000_000, "cache": 4_000_000, "batch": 2_000_000, "dim": 128,
         "zipf": 1.2, "type": "fp32"},
        # gradients of a small odd batch, rows of an odd width; the caller does not say how wide the ids are
        {"name": "aggregate_12k", "kind": "aggregate", "ids": 1_000_000, "n": 12_345, "dim": 47, "zipf": 1.1, "bits": False},
        # one trainer's share of the local aggregation over a table of 1e8 rows
        {"name": "aggregate_524k", "kind": "aggregate", "ids": 100_000_000, "n": 524_288, "dim": 128, "zipf": 1.2,
         "bits": True},
        # an owner's update from an unsorted list (all-to-all exchange), ids of unstated width
        {"name": "update_adam_60k", "kind": "update", "nodes": 20_000_000, "n": 60_000, "dim": 128, "zipf": 1.2,
         "type": "fp32", "optimizer": "adam", "slabs": False, "bits": False},
        # one eighth of a 240 M x 64 fp16 table, sorted slabs from 8 senders with 1,048,576 rows among them
        {"name": "update_adagrad_1m", "kind": "update", "nodes": 240_000_000, "n": 1_048_576, "dim": 64, "zipf": 1.1,
         "type": "fp16", "optimizer": "adagrad", "slabs": True, "bits": True},
        # the cold cache of a trainer: per-node flush periods from hotness
        {"name": "cold_100k", "kind": "cold", "nodes": 5_000_000, "cache": 500_000, "n": 100_000, "dim": 128, "zipf": 1.1},
        # the index as the reference's host code calls it
        {"name": "index_65k", "kind": "index", "nodes": 1_000_000, "cache": 100_000, "n": 65_536, "new": 8_192, "zipf": 1.1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "fetch", "fetch", "aggregate", "aggregate", "update", "update", "cold", "index"))
    zipf = round(rng.uniform(1.05, 1.3), 3)
    dim = rng.choice(DIMS)
    if kind == "step":
        nodes = _log_int(rng, 100_000, 20_000_000 * 128 // max(dim, 128))
        graph = rng.random() < 0.25
        return {"kind": kind, "nodes": nodes, "cache": int(nodes * rng.uniform(0.03, 0.2)),
                "batch": _log_int(rng, 1_000, 1_000_000 * 128 // max(dim, 128)), "dim": dim, "zipf": zipf,
                "optimizer": rng.choice(("adam", "adagrad")), "graph": graph,
                "ids": "gpu" if graph else rng.choice(("gpu", "host"))}
    if kind == "fetch":
        name = rng.choice(("fp32", "fp32", "fp32", "fp16", "fp64"))
        width = max(dim * torch.empty(0, dtype=TYPES[name]).element_size(), 512)
        nodes = _log_int(rng, 100_000, 20_000_000 * 512 // width)
        return {"kind": kind, "nodes": nodes, "cache": int(nodes * rng.uniform(0.03, 0.2)),
                "batch": _log_int(rng, 250, 2_000_000 * 512 // width), "dim": dim, "zipf": zipf, "type": name}
    if kind == "aggregate":
        dim = rng.choice(DIMS + (47,))
        return {"kind": kind, "ids": _log_int(rng, 10_000, 100_000_000), "n": _log_int(rng, 500, 1_000_000 * 128 // max(dim, 128)),
                "dim": dim, "zipf": zipf, "bits": rng.random() < 0.5}
    if kind == "update":
        return {"kind": kind, "nodes": _log_int(rng, 1_000_000, 100_000_000 * 64 // max(dim, 64)),
                "n": _log_int(rng, 2_000, 1_000_000 * 64 // max(dim, 64)), "dim": dim, "zipf": zipf,
                "type": rng.choice(("fp32", "fp32", "fp16")), "optimizer": rng.choice(("adam", "adagrad")),
                "slabs": rng.random() < 0.5, "bits": rng.random() < 0.5}
    nodes = _log_int(rng, 100_000, 5_000_000)
    cache = int(nodes * rng.uniform(0.03, 0.2))
    if kind == "cold":
        return {"kind": kind, "nodes": nodes, "cache": cache, "n": _log_int(rng, 1_000, max(nodes // 20, 1_000)), "dim": dim, "zipf": zipf}
    n = _log_int(rng, 500, 200_000)
    return {"kind": kind, "nodes": nodes, "cache": cache, "n": n, "new": max(n // 8, 1), "zipf": zipf}


# ---- ids ------------------------------------------------------------------------------------------------------------
def _ranks(gen, n, num, s, first=0):
    """n popularity ranks from [first, num), a power law by the inverse of its continuous distribution function."""
    u = torch.rand(n, dtype=torch.float64, device=gen.device, generator=gen)
    a, b = (first + 1.0) ** (1 - s), (num + 1.0) ** (1 - s)
    return ((a + u * (b - a)) ** (1 / (1 - s))).to(torch.int64).sub_(1).clamp_(first, num - 1)


def _rank_to_id(ranks, num):
    """``synth.rank_to_id`` on the GPU (its 64-bit products wrap in int64 as they do in uint64)."""
    k = max(int(num - 1).bit_length(), 2)
    mask, s1, s2 = (1 << k) - 1, max(k // 2, 1), max(k // 3, 1)
    m1, m2 = 0x9E3779B97F4A7C15 - (1 << 64), 0xD6E8FEB86659FD93 - (1 << 64)

    def mix(x):
        x = (x * m1) & mask
        x = x ^ (x >> s1)
        x = (x * m2) & mask
        x = x ^ (x >> s2)
        x = (x * m1) & mask
        return x ^ (x >> s1)

    out = mix(ranks)
    bad = out >= num
    while bool(bad.any()):
        out = torch.where(bad, mix(out), out)
        bad = out >= num
    return out


def _distinct_ids(gen, n, num, s, first=0):
    """About n distinct ids in no order, drawn by popularity."""
    r = torch.unique(_ranks(gen, 4 * n, num, s, first))
    if r.numel() > n:
        r = r[torch.randperm(r.numel(), device=gen.device, generator=gen)[:n]]
    return _rank_to_id(r[torch.randperm(r.numel(), device=gen.device, generator=gen)], num)


def _few_distinct(gen, n, num, s):
    """n ids by popularity, of which a number are distinct that n, num and s alone decide (results then have one shape
    whatever the seed): four deviations below the expected number; the rarest beyond it become the most popular."""
    r = _ranks(gen, n, num, s)
    seen = torch.unique(r)
    keep = max(int(_distinct(n, num, s) - 4 * math.sqrt(_distinct(n, num, s)) - 8), 1)
    return _rank_to_id(torch.where(r > seen[min(keep, seen.numel()) - 1], seen[0], r), num)


def _frontier(cfg, gen):
    """``synth.rmat_frontier`` on the GPU: the seeds and their sampled 1-hop and 2-hop neighbours."""
    layer = torch.randint(0, cfg.num_nodes, (cfg.seeds,), device=gen.device, generator=gen)
    parts = [layer]
    p0_s0, p0_s1 = cfg.a / (cfg.a + cfg.b), cfg.c / (1.0 - cfg.a - cfg.b)
    for fanout in cfg.fanout:
        u = layer.repeat_interleave(fanout)
        layer = torch.full_like(u, -1)
        while True:
            todo = layer < 0
            if not bool(todo.any()):
                break
            v = torch.zeros_like(u)
            for level in range(cfg.bits - 1, -1, -1):
                p0 = torch.where(((u >> level) & 1) == 0, p0_s0, p0_s1)
                v |= (torch.rand(u.shape, device=gen.device, generator=gen) >= p0).to(torch.int64) << level
            layer = torch.where(todo & (v < cfg.num_nodes), v, layer)
        parts.append(layer)
    return torch.cat(parts)


def _gen(seed, device="cuda"):
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    return gen


def _normal(gen, shape, sigma, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, device=gen.device).normal_(0.0, sigma, generator=gen)


# ---- what a user's program has in hand --------------------------------------------------------------------------------
def prepare(case, seed):
    st = {"step": _prepare_step, "fetch": _prepare_fetch, "aggregate": _prepare_aggregate, "update": _prepare_update,
          "cold": _prepare_cold, "index": _prepare_index}[case["kind"]](case, seed)
    st.kind, st.turn = case["kind"], getattr(st, "turn", 0)
    return st


def _next(st, items):
    """Programs come with new ids on every call: the prepared batches take turns."""
    st.turn += 1
    return items[(st.turn - 1) % len(items)]


def _prepare_step(case, seed):
    gen = _gen(seed)
    dim, batch = case["dim"], case["batch"]
    if "rmat_bits" in case:
        cfg = synth.scaled_rmat(synth.CONFIG5, case["rmat_bits"], case["seeds"])
        path = pipeline.build_rmat_path(cfg, optimizer=case["optimizer"])
        batches = [_frontier(cfg, gen) for _ in range(FLUSH_EVERY)]
    else:
        cfg = synth.CacheFetchConfig("perf_step", 1, case["nodes"], dim, case["cache"], batch, case["zipf"], flush_every=FLUSH_EVERY)
        path = pipeline.build_path(cfg, optimizer=case["optimizer"])
        batches = [_rank_to_id(_ranks(gen, batch, case["nodes"], case["zipf"]), case["nodes"]) for _ in range(FLUSH_EVERY)]
    grads = _normal(gen, (batch, dim), cfg.grad_sigma)
    st = SimpleNamespace(path=path, grads=grads, graph=case["graph"])
    opt, remote = path.opt, path.cold.remote
    st.buffers = {"table": path.table, "cache_rows": path.cold.emb, "staged": remote.grad, "staged_cnt": remote.cnt,
                  "staged_ids": remote.idx, "staged_age": remote.iter_count, "dropped": path.cold.dropped}
    st.buffers.update({k: v for k, v in vars(opt).items() if isinstance(v, torch.Tensor)})
    if case["graph"]:
        # as the repository's benchmark sets the path up
        path.want_locs, path.overlap_fetch = False, True
        st.batches, st.ids = batches, torch.empty(batch, dtype=torch.int64, device="cuda")
        st.rows = torch.empty((batch, dim), device="cuda")
    else:
        # a frontier has another length in every step
        st.batches = [b[: batch - (k * batch) // 400] for k, b in enumerate(batches)]
        if case["ids"] == "host":
            st.batches = [b.cpu().pin_memory() for b in st.batches]
        st.layer = DistEmb(path)
        st.sparse = DistembSparseGradOptimizer([st.layer.sparse_emb])
    st.turn = 0
    if case["graph"]:
        for _ in range(WARM_STEPS):
            st.ids.copy_(_next(st, st.batches))
            path.step(st.ids, grads, st.rows)
        torch.cuda.synchronize()
        path.capture(st.ids, grads, st.rows)
    else:
        for _ in range(WARM_STEPS):
            _run_step(st)
    return st


def _prepare_fetch(case, seed):
    gen = _gen(seed)
    nodes, dtype = case["nodes"], TYPES[case["type"]]
    table = _normal(gen, (nodes, case["dim"]), 0.01, dtype)
    index = E.IndexCache(case["cache"], "perf_fetch", True, False)
    hot = _rank_to_id(torch.arange(case["cache"], device="cuda"), nodes)
    slots = index.cuda_add(hot)
    rows = torch.zeros((index.get_capacity(), case["dim"]), dtype=dtype, device="cuda")
    rows[slots[slots >= 0]] = table[hot[slots >= 0]]
    batches = [_rank_to_id(_ranks(gen, case["batch"], nodes, case["zipf"]), nodes) for _ in range(4)]
    return SimpleNamespace(index=index, rows=rows, table=table, batches=batches)


def _prepare_aggregate(case, seed):
    gen = _gen(seed)
    batches = [(_few_distinct(gen, case["n"], case["ids"], case["zipf"]), _normal(gen, (case["n"], case["dim"]), 1e-3))
               for _ in range(4)]
    return SimpleNamespace(batches=batches, bits={"id_bits": _bits(case["ids"])} if case["bits"] else {})


def _bits(num_ids):
    return max(int(num_ids).bit_length() + 1, 8)


def _prepare_update(case, seed):
    gen = _gen(seed)
    nodes, dim, rank = case["nodes"], case["dim"], 3
    shard = ShardedEmbedding(nodes, dim, rank, SENDERS, dtype=TYPES[case["type"]], device=torch.device("cuda", torch.cuda.current_device()),
                             init_sigma=0.01, seed=seed)
    opt = (SparseAdam if case["optimizer"] == "adam" else SparseAdagrad)(shard, lr=0.01)
    batches = []
    for _ in range(2):
        # every sender has aggregated its own gradients: its ids are distinct; those of two senders overlap
        parts = [_distinct_ids(gen, case["n"] // SENDERS, shard.rows, case["zipf"]) * SENDERS + rank for _ in range(SENDERS)]
        if case["slabs"]:
            cap = max(p.numel() for p in parts)
            ids = torch.zeros((SENDERS, cap), dtype=torch.int64, device="cuda")
            for k, p in enumerate(parts):
                ids[k, : p.numel()] = p.sort().values
            ids = ids.flatten()
            how = {"seg_counts": torch.tensor([p.numel() for p in parts], device="cuda"), "seg_cap": cap, "sorted_segments": True}
        else:
            ids, how = torch.cat(parts), {}
        if case["bits"]:
            how["id_bits"] = _bits(nodes)
        cnt = torch.randint(1, 5, ids.shape, device="cuda", generator=gen)
        batches.append((ids, _normal(gen, (ids.numel(), dim), 1e-3), cnt, how))
    buffers = {"weight": shard.weight, **{k: v for k, v in vars(opt).items() if isinstance(v, torch.Tensor)}}
    return SimpleNamespace(opt=opt, batches=batches, buffers=buffers)


def _prepare_cold(case, seed):
    gen = _gen(seed)
    nodes, n = case["nodes"], case["n"]
    # flush periods from 1 round for the most popular cold ids to 25 for the rarest
    heat = torch.zeros(nodes, device="cuda")
    heat[_rank_to_id(torch.arange(nodes, device="cuda"), nodes)] = (0.01 * nodes / torch.arange(1, nodes + 1, device="cuda")).clamp(max=1.0) ** 0.7
    cache = ColdCache("perf_cold", case["cache"], case["dim"], threshold=flush_thresholds(heat), cnt_threshold=16)
    shard = ShardedEmbedding(nodes, case["dim"], init_sigma=0.01, seed=seed)
    opt = SparseAdagrad(shard, lr=0.01)
    batches = []
    for _ in range(4):
        ids = _distinct_ids(gen, n, nodes, case["zipf"], first=nodes // 100)
        batches.append((ids, _normal(gen, (ids.numel(), case["dim"]), 0.01), _normal(gen, (ids.numel(), case["dim"]), 1e-3)))
    r = cache.remote
    st = SimpleNamespace(cache=cache, opt=opt, batches=batches, turn=0,
                         buffers={"cache_rows": cache.emb, "staged": r.grad, "staged_cnt": r.cnt, "staged_ids": r.idx,
                                  "staged_age": r.iter_count, "dropped": cache.dropped, "weight": shard.weight,
                                  "state_sum": opt.state_sum})
    for _ in range(3):  # a cache in use holds rows of several rounds
        _run_cold(st)
    return st


def _prepare_index(case, seed):
    gen = _gen(seed)
    nodes = case["nodes"]
    index = E.IndexCache(case["cache"], "perf_index", True, False)
    index.cuda_add(_rank_to_id(torch.arange(case["cache"], device="cuda"), nodes))
    batches = [(_rank_to_id(_ranks(gen, case["n"], nodes, case["zipf"]), nodes).cpu(),
                _distinct_ids(gen, case["new"], nodes, case["zipf"], first=case["cache"]).cpu()) for _ in range(4)]
    return SimpleNamespace(index=index, batches=batches)


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(state):
    return {"step": _run_step, "fetch": _run_fetch, "aggregate": _run_aggregate, "update": _run_update, "cold": _run_cold,
            "index": _run_index}[state.kind](state)


def _run_step(st):
    ids = _next(st, st.batches)
    if st.graph:
        rows, _, found, stats = st.path.step(ids, st.grads, st.rows)
        return {"rows": rows, "found": found, "distinct": stats.num_unique, "classes": stats.split_counts, **st.buffers}
    rows = st.layer(ids)
    rows.grad = st.grads[: ids.numel()]  # what the model's backward pass leaves
    st.sparse.zero_grad()
    st.sparse.step()
    return {"rows": rows.detach(), **st.buffers}


def _run_fetch(st):
    rows, slots, found = E.cudaLookupFetch(st.index, _next(st, st.batches), st.rows, st.table)
    return {"rows": rows, "slots": slots, "found": found}


def _run_aggregate(st):
    ids, grads = _next(st, st.batches)
    unique, sums, counts = only_unique_grads(ids, grads, **st.bits)
    return {"ids": unique, "sums": sums, "counts": counts}


def _run_update(st):
    ids, grads, cnt, how = _next(st, st.batches)
    st.opt.update(ids, grads, cnt, **how)
    return st.buffers


def _run_cold(st):
    ids, rows, grads = _next(st, st.batches)
    slots = st.cache.insert(ids, rows)
    st.cache.accumulate_remote(ids, grads)
    out_ids, out_rows, out_cnt, counts = st.cache.flush_remote()
    st.opt.update(out_ids, out_rows, out_cnt, is_unique=True)
    return {"slots": slots, "left": counts, **st.buffers}


def _run_index(st):
    ids, new = _next(st, st.batches)
    slots = st.index.lookup(ids)
    return {"slots": slots, "new": st.index.add(new)}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _distinct(n, num, s, first=0, last=None):
    """Expected number of distinct ranks in [first, last) among n drawn from the power law over [0, num)."""
    last = num if last is None else last
    edges = np.unique(np.floor(np.geomspace(first + 1, last + 1, 4000)))
    whole = 1.0 - (num + 1.0) ** (1 - s)
    width = np.diff(edges)
    p = (edges[:-1] ** (1 - s) - edges[1:] ** (1 - s)) / whole / width
    return float(np.sum(width * -np.expm1(n * np.log1p(-np.minimum(p, 1 - 1e-12)))))


def work(case):
    kind = case["kind"]
    if kind == "index":
        n, new = case["n"], case["new"]
        return {"bytes": 16 * n + 16 * new + 12 * 8 * min(n, case["cache"] / 8), "flops": 0}
    dim = case["dim"]
    if kind == "step":
        n, row, d = case["batch"], 4 * dim, {}
        states = 2 if case["optimizer"] == "adam" else 1
        if "rmat_bits" in case:
            d = {"all": 0.62 * n, "hot": 0.3 * n, "cold": 0.32 * n, "flush": 2.1 * n}  # counted on such frontiers
        else:
            num, s, hot = case["nodes"], case["zipf"], case["nodes"] // 100
            d = {"all": _distinct(n, num, s), "hot": _distinct(n, num, s, 0, hot), "cold": _distinct(n, num, s, hot),
                 "flush": min(_distinct(FLUSH_EVERY * n, num, s, hot), case["cache"])}
        forward = 8 * n + n + row * (d["all"] + n)               # ids, found; each row once, the rows of the batch
        updates = d["hot"] + min(d["flush"], 1 << 19) / FLUSH_EVERY
        backward = row * (n + 2 * updates * (1 + states))         # gradients; weights and optimiser state
        staging = row * (2 * min(d["cold"], case.get("cache", n)) + 2 * min(d["flush"], 1 << 19) / FLUSH_EVERY)
        return {"bytes": forward + backward + staging, "flops": dim * (n + 12 * updates)}
    if kind == "fetch":
        n = case["batch"]
        row = dim * torch.empty(0, dtype=TYPES[case["type"]]).element_size()
        return {"bytes": n * (8 + 8 + 1 + row) + row * _distinct(n, case["nodes"], case["zipf"]), "flops": 0}
    n = case["n"]
    if kind == "aggregate":
        u = _distinct(n, case["ids"], case["zipf"])
        return {"bytes": n * (8 + 4 * dim) + u * (16 + 4 * dim), "flops": n * dim}
    if kind == "update":
        # each sender draws about its share of distinct rows: count those of all senders together
        u = 0.6 * n
        states = 2 if case["optimizer"] == "adam" else 1
        elem = 2 if case["type"] == "fp16" else 4
        return {"bytes": n * (16 + 4 * dim) + u * 2 * dim * (4 * states + elem), "flops": n * dim + 12 * u * dim}
    # cold: rows and gradients in; cached rows and staged rows; some 0.4 n rows leave: read, zeroed, weight and state updated
    return {"bytes": n * (8 + 4 * dim * (5 + 0.4 * 6)) + 16 * case["cache"], "flops": 3 * n * dim}


def tolerance(case):
    kind = case["kind"]
    if kind in ("fetch", "index"):
        return "exact"      # rows and whole numbers are copied
    if kind in ("step", "update", "cold"):
        # The first updates of a row are lr * g / |g|: where a sum of gradients nearly cancels, its last bit decides
        # over a whole update of a single value.  fp16 weights are off by one unit where a value lies between two.
        return {"rel": 1e-4, "max": 0.5}
    return {"rel": 1e-5}    # sums in fp32
