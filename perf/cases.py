"""The work a user of this library has it do, as measurable cases.

Every case goes through the public surface: torch.classes.dgs_classes.ChunkTensor, torch.ops.dgs_ops.* and
PipelinedSampler.  Six kinds:

  index     ChunkTensor._CAPI_index: rows of a feature / label table by id (optionally with a pinned host tail)
  cache     _CAPI_fetch_data_chunk_tensor: rows through the hash table of a cache, misses from pinned host memory
  hop       one hop of the reference's own loop: _CAPI_sample_neighbors* and _CAPI_tensor_relabel
  weighted  _CAPI_sample_neighbors_with_probs* (A-Res without, proportional draws with replacement)
  blocks    _CAPI_sample_blocks_with_chunk_tensor, then the feature rows of the input nodes
  pipeline  PipelinedSampler: mini-batches in flight, each with its feature rows

Sampling is random but reproducible: run() seeds torch's CUDA generator, as a program does that wants the same
mini-batch for the same step number.  Graphs are Chung-Lu power laws in CSC form, the seeds of a hop are a
frontier (nodes met by following random edges, so hubs are among them), the seeds of a batch are training nodes.
How many nodes a batch meets is decided by the draw; so that the outputs of two inputs can still be laid side by
side, the inputs of every seed are the same graph under another numbering of its nodes (another indptr, other
neighbour ids, other seeds, other features and weights), and the random stream is the one of the step.
"""
import importlib

import torch

pkg = importlib.import_module("dist-gpu-sampling_b200")
synth = importlib.import_module("dist-gpu-sampling_b200.synth")

DTYPES = {"float32": torch.float32, "float64": torch.float64, "int64": torch.int64, "int32": torch.int32,
          "bool": torch.bool}
ESZ = {"float32": 4, "float64": 8, "int64": 8, "int32": 4, "bool": 1}


def listed():
    return [
        # labels of one mini-batch: the smallest call there is, all latency
        dict(name="labels_of_a_batch", kind="index", rows=2_449_029, dim=1, n=1024, dtype="int64", ids="int64",
             gpu_share=1.0),
        # feature rows of one mini-batch's input nodes, the Products-shaped table
        dict(name="features_100", kind="index", rows=2_449_029, dim=100, n=430_000, dtype="float32", ids="int64",
             gpu_share=1.0),
        # the largest query: 0.8 GB out of a 4 GB table of wide rows
        dict(name="features_256_large", kind="index", rows=4_000_000, dim=256, n=800_000, dtype="float32",
             ids="int64", gpu_share=1.0),
        # a row width that is no multiple of 16 bytes
        dict(name="features_75_ragged", kind="index", rows=1_500_000, dim=75, n=333_333, dtype="float32",
             ids="int64", gpu_share=1.0),
        # hybrid placement: part of the table in pinned host memory, met by some of the ids
        dict(name="features_host_tail", kind="index", rows=1_000_000, dim=128, n=200_000, dtype="float32",
             ids="int64", gpu_share=0.9),
        # the cache operator: most rows hit, the others come from pinned host memory
        dict(name="cache_fetch", kind="cache", rows=400_000, dim=128, n=60_000, dtype="float32", ids="int64",
             hit=0.97),
        # the last hop of a Products-shaped batch, operator by operator
        dict(name="hop_60k_15", kind="hop", nodes=2_449_029, deg=50.5, seeds=60_000, fanout=15, ids="int64",
             replace=False, chunk=True),
        # second hop of a weighted [10, 10] batch on a hub-heavy graph
        dict(name="weighted_11k_10", kind="weighted", nodes=2_000_000, deg=55.0, seeds=11_000, fanout=10,
             ids="int64", replace=False, chunk=True),
        # proportional draws with replacement
        dict(name="weighted_replace_4k_10", kind="weighted", nodes=500_000, deg=30.0, seeds=4096, fanout=10,
             ids="int64", replace=True, chunk=True),
        # a small batch, as inference on a few nodes asks for: a chain of short launches
        dict(name="blocks_small", kind="blocks", nodes=500_000, deg=30.0, seeds=64, hops="10,5", dim=64,
             ids="int64"),
        # one training batch at a time
        dict(name="blocks_batch", kind="blocks", nodes=2_449_029, deg=50.5, seeds=1024, hops="15,10,5", dim=100,
             ids="int64"),
        # the headline workload: six training batches in flight
        dict(name="pipeline_batches", kind="pipeline", nodes=2_449_029, deg=50.5, seeds=1024, hops="15,10,5",
             dim=100, ids="int64"),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["index", "index", "index", "cache", "hop", "weighted", "blocks", "pipeline"])
    ids = rng.choice(["int64", "int64", "int32"])
    if kind == "index":
        dtype = rng.choice(["float32", "float32", "float32", "float64", "int64", "bool"])
        dim = 1 if rng.random() < 0.15 else _log(rng, 3, 256)
        if dtype in ("float64", "int64"):
            dim = max(1, dim // 2)
        return dict(kind=kind, rows=_log(rng, 50_000, 4_000_000), dim=dim, n=_log(rng, 300, 800_000), dtype=dtype,
                    ids=ids, gpu_share=0.9 if rng.random() < 0.2 else 1.0)
    if kind == "cache":
        return dict(kind=kind, rows=_log(rng, 50_000, 400_000), dim=_log(rng, 8, 256), n=_log(rng, 1000, 60_000),
                    dtype="float32", ids=ids, hit=rng.choice([0.9, 0.97, 0.99]))
    if kind == "hop":
        return dict(kind=kind, nodes=_log(rng, 100_000, 2_449_029), deg=round(rng.uniform(8.0, 50.0), 1),
                    seeds=_log(rng, 256, 60_000), fanout=rng.choice([5, 10, 15, 25]), ids=ids,
                    replace=rng.random() < 0.25, chunk=rng.random() < 0.7)
    if kind == "weighted":
        replace = rng.random() < 0.4
        return dict(kind=kind, nodes=_log(rng, 100_000, 500_000 if replace else 2_000_000),
                    deg=round(rng.uniform(8.0, 30.0 if replace else 55.0), 1),
                    seeds=_log(rng, 256, 4096 if replace else 11_000), fanout=rng.choice([5, 10, 15, 25]), ids=ids,
                    replace=replace, chunk=rng.random() < 0.7)
    hops = rng.choice(["15,10,5", "10,10", "10,5", "25,10"])
    return dict(kind=kind, nodes=_log(rng, 200_000, 2_449_029), deg=round(rng.uniform(10.0, 50.0), 1),
                seeds=_log(rng, 16, 1024), hops=hops, dim=_log(rng, 16, 128), ids=ids)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _chunk(t, gpu_share=1.0):
    """A ChunkTensor that holds `t` (on the GPU); the rows beyond gpu_share of them in the pinned host tail."""
    rows = t.shape[0]
    row_bytes = t.element_size() * (t.numel() // max(rows, 1))
    keep = rows if gpu_share >= 1.0 else int(rows * gpu_share) // 16 * 16
    ct = torch.classes.dgs_classes.ChunkTensor(list(t.shape), t.dtype, max(keep * row_bytes, 1))
    flat = t.reshape(-1)
    sub = ct._CAPI_get_sub_device_tensor()
    sub[:min(sub.numel(), flat.numel())].copy_(flat[:sub.numel()])
    host = ct._CAPI_get_host_tensor()
    if host.numel():
        host.copy_(flat[flat.numel() - host.numel():].cpu())
    return ct, keep


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _table(rows, dim, dtype, g):
    shape = (rows,) if dim == 1 else (rows, dim)
    if dtype == "bool":
        return torch.randint(0, 2, shape, device="cuda", generator=g, dtype=torch.uint8).to(torch.bool)
    if dtype in ("int64", "int32"):
        return torch.randint(0, 1 << 20, shape, device="cuda", generator=g, dtype=DTYPES[dtype])
    return torch.randn(shape, device="cuda", generator=g, dtype=DTYPES[dtype])


STEP = 11  # the step whose mini-batch is drawn: the random stream of every pass


def _renumber(indptr, indices, new_id):
    """The same CSC graph with node v called new_id[v]; the neighbours of a row keep their order."""
    old = torch.argsort(new_id)
    deg = (indptr[1:] - indptr[:-1])[old]
    out = torch.zeros_like(indptr)
    torch.cumsum(deg, 0, out=out[1:])
    at = torch.repeat_interleave(indptr[:-1][old] - out[:-1], deg)
    at += torch.arange(at.numel(), device="cuda")
    return out, new_id[indices[at]]


def _frontier(indices, n, g):
    """n distinct nodes met by following random edges, in random order."""
    have = torch.empty(0, dtype=indices.dtype, device="cuda")
    while have.numel() < n:
        pick = torch.randint(0, indices.numel(), (2 * n,), device="cuda", generator=g)
        have = torch.unique(torch.cat([have, indices[pick]]))
    return have[torch.randperm(have.numel(), device="cuda", generator=g)[:n]].contiguous()


def _hops(case):
    return [int(k) for k in case["hops"].split(",")]


BATCHES = 6  # of a pipeline pass; as many are in flight


def _index_inputs(case, seed):
    """(table, ids) of an index case: ids as a frontier's, distinct and in no order."""
    g = _gen(seed)
    table = _table(case["rows"], case["dim"], case["dtype"], g)
    if case["n"] <= case["rows"]:
        ids = torch.randperm(case["rows"], device="cuda", generator=g)[:case["n"]]
    else:
        ids = torch.randint(0, case["rows"], (case["n"],), device="cuda", generator=g)
    return table, ids.to(DTYPES[case["ids"]])


def _cache_inputs(case, seed):
    """(table, cached row numbers, asked ids): three quarters of the rows are cached, `hit` of the ids are met."""
    g = _gen(seed)
    rows, n = case["rows"], case["n"]
    table = _table(rows, case["dim"], case["dtype"], g)
    perm = torch.randperm(rows, device="cuda", generator=g)
    cached, rest = perm[:rows * 3 // 4], perm[rows * 3 // 4:]
    hits = min(int(n * case["hit"]), cached.numel())
    misses = min(n - hits, rest.numel())
    ids = torch.cat([cached[torch.randperm(cached.numel(), device="cuda", generator=g)[:hits]], rest[:misses]])
    return table, cached, ids[torch.randperm(ids.numel(), device="cuda", generator=g)]


def prepare(case, seed):
    pkg.load_ops()
    torch.cuda.init()
    kind = case["kind"]
    state = {"kind": kind, "generator": torch.cuda.default_generators[torch.cuda.current_device()]}
    if kind == "index":
        table, ids = _index_inputs(case, seed)
        state["table"], _ = _chunk(table, case["gpu_share"])
        state["ids"] = ids
        return state
    if kind == "cache":
        table, cached, ids = _cache_inputs(case, seed)
        idt = DTYPES[case["ids"]]
        state["host"] = table.cpu().pin_memory()
        state["gpu"], _ = _chunk(table[cached])
        state["keys"], state["values"] = torch.ops.dgs_ops._CAPI_create_hash_map(
            cached.to(idt), torch.arange(cached.numel(), device="cuda", dtype=idt))
        state["ids"] = ids.to(idt)
        return state
    idt = DTYPES[case["ids"]]
    indptr, indices = synth.chung_lu_csc(case["nodes"], case["deg"], 2.1, seed=STEP, device="cuda")
    step, g = _gen(STEP), _gen(seed)
    if kind in ("hop", "weighted"):
        batches = [_frontier(indices, min(case["seeds"], case["nodes"] // 8), step)]
    else:
        batches = [torch.randperm(case["nodes"], device="cuda", generator=step)[:case["seeds"]]
                   for _ in range(BATCHES if kind == "pipeline" else 1)]
    new_id = torch.randperm(case["nodes"], device="cuda", generator=g)
    indptr, indices = _renumber(indptr, indices, new_id)
    indptr, indices = indptr.to(idt), indices.to(idt)
    batches = [new_id[b].to(idt) for b in batches]
    if kind in ("hop", "weighted"):
        state["seeds"] = batches[0]
        state["fanout"], state["replace"], state["chunk"] = case["fanout"], case["replace"], case["chunk"]
        probs = torch.rand(indices.numel(), device="cuda", generator=g) if kind == "weighted" else None
        if case["chunk"]:
            state["indptr"], state["indices"] = _chunk(indptr)[0], _chunk(indices)[0]
            state["probs"] = _chunk(probs)[0] if probs is not None else None
        else:
            state["indptr"], state["indices"], state["probs"] = indptr, indices, probs
        return state
    state["indptr"], state["indices"] = _chunk(indptr)[0], _chunk(indices)[0]
    state["features"] = _chunk(_table(case["nodes"], case["dim"], "float32", g))[0]
    state["hops"] = _hops(case)
    if kind == "blocks":
        state["seeds"] = batches[0]
    else:
        state["batches"] = batches
        state["sampler"] = pkg.PipelinedSampler(state["indptr"], state["indices"], state["hops"],
                                                features=state["features"], max_seeds=case["seeds"], depth=BATCHES)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    ops = torch.ops.dgs_ops
    if kind == "index":
        return state["table"]._CAPI_index(state["ids"])
    if kind == "cache":
        return ops._CAPI_fetch_data_chunk_tensor(state["host"], state["gpu"], state["ids"], state["keys"],
                                                 state["values"])
    state["generator"].manual_seed(STEP)
    if kind == "hop":
        fn = ops._CAPI_sample_neighbors_with_chunk_tensor if state["chunk"] else ops._CAPI_sample_neighbors
        row, col = fn(state["seeds"], state["indptr"], state["indices"], state["fanout"], state["replace"])
        frontier, (row, col) = ops._CAPI_tensor_relabel([state["seeds"], col], [row, col])
        return frontier, row, col
    if kind == "weighted":
        fn = ops._CAPI_sample_neighbors_with_probs_with_chunk_tensor if state["chunk"] \
            else ops._CAPI_sample_neighbors_with_probs
        return fn(state["seeds"], state["indptr"], state["indices"], state["probs"], state["fanout"],
                  state["replace"])
    if kind == "blocks":
        frontier, blocks, _ = pkg.sample_blocks(state["seeds"], state["hops"], state["indptr"], state["indices"],
                                                fused=True)
        return frontier, [b[:2] for b in blocks], state["features"]._CAPI_index(frontier)
    for seeds in state["batches"]:
        state["sampler"].submit(seeds)
    out = []
    for _ in state["batches"]:
        frontier, blocks, _, x = state["sampler"].next()
        out.append((frontier, [b[:2] for b in blocks], x))
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _block_bytes(case):
    """Seeds, row bounds, picked neighbours read once; rows, columns and frontiers written once; feature rows
    read and written.  The sizes that the draw decides are taken as: every seed of mean degree or more fills its
    fan-out, and a hop finds new nodes until about two thirds of those within reach are met."""
    e = ESZ[case["ids"]]
    n, total = min(case["seeds"], case["nodes"]), 0
    for k in reversed(_hops(case)):
        edges = n * min(k, 0.9 * case["deg"])
        new = min(edges, case["nodes"] * 0.66 * edges / (edges + case["nodes"]))
        total += 3 * e * n + 3 * e * edges + e * (n + new)
        n += new
    return total + n * (e + 2 * 4 * case["dim"])


def work(case):
    kind, e = case["kind"], ESZ[case["ids"]]
    if kind in ("index", "cache"):
        return {"bytes": case["n"] * (e + 2 * case["dim"] * ESZ[case["dtype"]]), "flops": 0}
    if kind in ("hop", "weighted"):
        n = min(case["seeds"], case["nodes"] // 8)
        edges = n * (case["fanout"] if case["replace"] else min(case["fanout"], 2 * case["deg"]))
        total = 3 * e * n + 3 * e * edges
        if kind == "hop":      # the relabel reads seeds, rows and columns and writes rows, columns and the frontier
            total += e * n + 4 * e * edges + e * (n + 0.5 * edges)
        else:                  # every weight of a row decides; rows met along edges are 11 to 15 times the mean
            total += 4 * n * 13 * case["deg"]
        return {"bytes": total, "flops": 0}
    return {"bytes": _block_bytes(case) * (BATCHES if kind == "pipeline" else 1), "flops": 0}


def tolerance(case):
    # Rows, ids and labels are whole numbers or copied bytes.  Only the proportional draws come out of float sums:
    # prefix sums of fp32 weights taken in two orders (windows of 32 and of 512, rows of 50 to 12,000 weights) put
    # 2.6e-4 of the draws on the neighbouring edge; four times that.
    if case["kind"] == "weighted" and case["replace"]:
        return {"rel": 0.0, "differ": 1e-3}
    return "exact"


def exact(case, seed):
    # copied rows are what float outputs there are; sampled blocks are whole numbers around the same copy
    if case["kind"] == "index":
        table, ids = _index_inputs(case, seed)
        out = table.reshape(case["rows"], -1)[ids.long()]
        return out.double() if out.is_floating_point() else None
    if case["kind"] == "cache":
        table, _, ids = _cache_inputs(case, seed)
        return table[ids].double()
    return None
