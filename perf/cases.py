"""Workloads of the minibatch path, sized for timing: sampling with feature gather (one
batch at a time, prefetching loaders, the epoch driver, heterogeneous graphs), the plain
feature gathers and the one-hop Philox sampler.

A case is a dict of plain values.  `prepare` builds what a training program holds before it
asks for batches (graph and features in HBM, seed ids, the sampler or loader object), `run`
makes one pass through the public API, `work` states the bytes the pass cannot do without.
Graphs are R-MAT (skewed degrees, duplicate edges, isolated vertices) and seeds are uniform,
like the repository's benchmark.  All results are integers or exact decodes of stored
values, so every output is compared bit for bit.

How many vertices a batch reaches depends on every vertex id, weight and draw, so inputs of
another seed are the same graph under other vertex names (`permute` keeps the order within
a row, and the reference's random stream names row positions), other seed ids to match, and
other feature rows: batches of the same shape out of other values at other addresses.
Where the result does depend on the names (Philox draws, sorted typed adjacencies) the
feature rows alone are new.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import aethergraph_b200 as ag
from aethergraph_b200 import synth
from aethergraph_b200.pytorch import NeighborLoader as EpochLoader
from aethergraph_b200.sampler import reservoir_hop

DTYPES = ("f32", "f16", "bf16", "i8")
GRAPH_SEED, SEEDS_SEED, SAMPLER_SEED = 1, 3, 42
ELEMENT = {"f32": 4, "f16": 2, "bf16": 2, "i8": 1}


def _sampling(name, kind, **kw):
    case = dict(name=name, kind=kind, nodes=1 << 20, edges=16 << 20, dim=128, dtype="f32", batch=128, batches=1,
                fanout="15,10", replace=False, weighted=False, rng="wyrand_exact", subgraph="directional",
                edge_ids=True, threads=1, group=8, depth=2)
    case.update(kw)
    return case


def listed():
    return [
        # Online inference on a medium graph: one small batch, answered before the next is asked for.
        _sampling("sample_b128", "sample"),
        # The same call with a training-size batch over a table of feature rows far larger than L2.
        _sampling("sample_b1024", "sample", nodes=1 << 24, edges=320_000_000, dim=256, dtype="bf16", batch=1024,
                  fanout="25,10"),
        # Subgraph methods that keep every edge between the sampled vertices.
        _sampling("sample_induced_b200", "sample", nodes=4_000_000, edges=64_000_000, dim=100, dtype="f16", batch=200,
                  fanout="10,5", subgraph="induced"),
        # `for batch in loader` with the epoch driver's defaults over a small training split, ragged last batch.
        _sampling("epoch_b128", "epoch", batches=10, inputs=1200, depth=3),
        # Prefetching loader feeding a training loop: large batches, two sampler threads.
        _sampling("loader_b1024", "loader", nodes=1 << 24, edges=320_000_000, dim=256, dtype="bf16", batch=1024, batches=12,
                  fanout="25,10", threads=2, depth=12),
        # Importance-weighted edges, three hops.
        _sampling("loader_weighted_b512", "loader", nodes=10_000_000, edges=200_000_000, dim=128, dtype="f16", batch=512,
                  batches=12, fanout="15,10,5", weighted=True, threads=2, depth=12),
        # Deep neighborhoods of very large batches: the largest subgraphs the path is used for.
        _sampling("loader_3hop_b4096", "loader", nodes=20_000_000, edges=480_000_000, dim=128, dtype="bf16", batch=4096,
                  batches=6, fanout="15,10,5", threads=2, group=4, depth=6),
        # Block-scaled int8 rows, a ragged batch size.
        _sampling("loader_int8_b777", "loader", nodes=3_000_000, edges=60_000_000, dim=160, dtype="i8", batch=777, batches=12,
                  fanout="10,10", threads=2, depth=12),
        # Typed graph (users, posts, comments, subreddits; six relations), rows of every type.
        dict(name="hetero_loader_b1024", kind="hetero", users=5_000_000, dim=128, dtype="bf16", batch=1024, batches=4,
             fanout="15,10/10,5/3,2", replace=False, rng="wyrand_exact", threads=2, group=4, depth=4),
        # Rows of a large id list, e.g. layer-wise inference over all vertices in a shuffled order.
        dict(name="gather_bf16", kind="gather", nodes=10_000_000, dim=256, dtype="bf16", rows=1_000_000, ids="int64"),
        # Rows that are not a whole number of 16-byte vectors.
        dict(name="gather_f16_d100", kind="gather", nodes=4_000_001, dim=100, dtype="f16", rows=200_003, ids="int32"),
        # Rows for a host-side consumer: ids and result in host memory.
        dict(name="get_batch_host", kind="get_batch", nodes=1 << 20, dim=128, dtype="f32", rows=20_000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_sampling(rng):
    kind = rng.choice(["sample", "sample", "loader", "loader", "epoch"])
    fanout = rng.choice(["15,10", "25,10", "10,5", "10,10", "15,10,5", "5,5,5", "20", "40,10", "8,4"])
    reach = 1
    for k in reversed(fanout.split(",")):
        reach = 1 + int(k) * reach
    batch = min(_log_uniform(rng, 16, 4096), max(16, 2_000_000 // reach))
    nodes = _log_uniform(rng, 1 << 16, 14_000_000)
    mode = rng.choice(["uniform"] * 5 + ["replace", "weighted", "weighted"])
    case = _sampling("", kind, nodes=nodes, edges=nodes * rng.randint(8, 24), dim=rng.choice([16, 50, 64, 100, 128, 200, 256, 301]),
                     dtype=rng.choice(DTYPES), batch=batch, fanout=fanout, replace=mode == "replace",
                     weighted=mode == "weighted", rng=rng.choice(["wyrand_exact", "wyrand_exact", "philox"]),
                     subgraph=rng.choice(["directional"] * 5 + ["bidirectional", "induced"]) if batch <= 512 else "directional",
                     edge_ids=rng.random() < 0.8, threads=rng.randint(1, 2), group=rng.choice([4, 8, 16]))
    if kind == "loader":
        case.update(batches=rng.randint(2, 12), depth=rng.choice([2, 4, 12]))
        while case["batches"] * batch * reach > 8_000_000:
            case["batches"] -= 1
    elif kind == "epoch":
        case.update(batches=rng.randint(2, 10), depth=3)
        while case["batches"] * batch * reach > 8_000_000:
            case["batches"] -= 1
        case["inputs"] = case["batches"] * batch - rng.randint(0, batch - 1)
    del case["name"]
    return case


def draw(rng):
    while True:
        case = _draw(rng)
        if work(case)["bytes"] <= 1_500_000_000:  # no larger than the largest listed case
            return case


def _draw(rng):
    kind = rng.choice(["sampling"] * 5 + ["hetero", "gather", "gather", "get_batch", "hop"])
    if kind == "sampling":
        return _draw_sampling(rng)
    if kind == "hetero":
        return dict(kind="hetero", users=_log_uniform(rng, 100_000, 5_000_000), dim=rng.choice([64, 100, 128]),
                    dtype=rng.choice(DTYPES), batch=_log_uniform(rng, 32, 1024), batches=rng.randint(1, 4),
                    fanout=rng.choice(["15,10/10,5/3,2", "10,5/5,5/2,2", "8,8/8,4/1,1"]), replace=rng.random() < 0.2,
                    rng=rng.choice(["wyrand_exact", "wyrand_exact", "philox"]), threads=rng.randint(1, 2),
                    group=rng.choice([1, 4, 8]), depth=rng.choice([2, 4]))
    if kind == "hop":
        nodes = _log_uniform(rng, 1 << 16, 1 << 22)
        return dict(kind="hop", nodes=nodes, edges=nodes * rng.randint(8, 24), rows=_log_uniform(rng, 100, 300_000),
                    fanout=rng.choice([5, 10, 15, 25, 40]))
    dim = rng.choice([1, 16, 33, 64, 100, 128, 200, 256, 301, 602, 768])
    dtype = rng.choice(DTYPES)
    nodes = _log_uniform(rng, 10_000, 5_000_000)
    if kind == "get_batch":
        return dict(kind="get_batch", nodes=nodes, dim=dim, dtype=dtype, rows=_log_uniform(rng, 1, max(2, 8_000_000 // dim)))
    return dict(kind="gather", nodes=nodes, dim=dim, dtype=dtype, rows=_log_uniform(rng, 32, max(64, 200_000_000 // dim)),
                ids=rng.choice(["int64", "int32"]))


# ------------------------------------------------------------------ prepare --
def _fanouts(text):
    return [int(k) for k in text.split(",")]


def _store(nodes, dim, dtype, seed):
    if dtype != "i8":
        return synth.features(nodes, dim, dtype, seed)
    g = torch.Generator("cuda").manual_seed(seed)
    return ag.FeatureStore.from_array(torch.randn(nodes, dim, device="cuda", generator=g), "i8")


HETERO_RELATIONS = (("user", "votes", "post"), ("user", "writes", "comment"), ("post", "belongs_to", "subreddit"),
                    ("post", "rev_votes", "user"), ("comment", "rev_writes", "user"), ("subreddit", "rev_belongs_to", "post"))


def _hetero_sizes(users):
    return {"user": users, "post": max(1, users * 2 // 5), "comment": users * 2, "subreddit": max(1, users // 500)}


def _hetero_graph(users):
    """user-votes-post (out-degree 30), user-writes-comment (8), post-belongs_to-subreddit (1) and their reverses."""
    n = _hetero_sizes(users)
    votes = synth.rmat_relation(n["user"], n["post"], 30 * users, GRAPH_SEED)
    writes = synth.rmat_relation(n["user"], n["comment"], 8 * users, GRAPH_SEED + 1)
    g = torch.Generator("cuda").manual_seed(GRAPH_SEED + 2)
    where = torch.randint(n["subreddit"], (n["post"],), device="cuda", dtype=torch.int32, generator=g)
    forward = [(synth.relation_sources(votes[0]), votes[1]), (synth.relation_sources(writes[0]), writes[1]),
               (torch.arange(n["post"], dtype=torch.int32, device="cuda"), where)]
    pairs = forward + [(b, a) for a, b in forward]
    return ag.HeteroCsrGraph.from_device_edges(n, [(*r, *p) for r, p in zip(HETERO_RELATIONS, pairs)])


def _graph(case, seed):
    """The case's graph under vertex names of its own, and the function from the first names to those."""
    n = case["nodes"]
    graph = synth.rmat_graph(n, case["edges"], GRAPH_SEED, weight_sigma=1.0 if case["weighted"] else 0.0)
    if case["rng"] == "philox":
        return graph, lambda ids: ids
    r = np.random.default_rng(seed)
    a, b = int(r.integers(1, n)), int(r.integers(n))
    while math.gcd(a, n) != 1:
        a += 1
    first_name = (torch.arange(n, device="cuda") * a + b) % n
    back = pow(a, -1, n)
    return (graph.permute(first_name.to(torch.int32).cpu().numpy()),
            lambda ids: ((np.asarray(ids, dtype=np.int64) - b) % n * back % n).astype(np.uint32))


def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "hetero":
        s["graph"] = graph = _hetero_graph(case["users"])
        torch.cuda.empty_cache()
        sizes = _hetero_sizes(case["users"])
        stores = {t: _store(sizes[t], 64 if t == "subreddit" else case["dim"], case["dtype"], seed + 10 + i)
                  for i, t in enumerate(sizes)}
        fan = [_fanouts(f) for f in case["fanout"].split("/")] * 2
        cfg = ag.HeteroSamplingConfig(dict(zip(HETERO_RELATIONS, fan)), replace=case["replace"], seed=SAMPLER_SEED,
                                      rng_mode=case["rng"])
        s["seeds"] = [synth.seed_batch(case["users"], case["batch"], SEEDS_SEED, b) for b in range(case["batches"])]
        if case["batches"] == 1:
            s["sampler"] = ag.HeteroNeighborSampler(graph, cfg, features=stores)
        else:
            s["loader"] = ag.HeteroNeighborLoader(graph, cfg, "user", prefetch_depth=case["depth"], features=stores,
                                                  sampler_threads=case["threads"], group=case["group"])
        return s
    if kind in ("gather", "get_batch"):
        s["store"] = _store(case["nodes"], case["dim"], case["dtype"], seed)
        if kind == "get_batch":
            s["ids"] = np.random.default_rng(seed).integers(0, case["nodes"], case["rows"])
        else:
            g = torch.Generator("cuda").manual_seed(seed + 1)
            s["ids"] = torch.randint(case["nodes"], (case["rows"],), device="cuda", generator=g,
                                     dtype=torch.int64 if case["ids"] == "int64" else torch.int32)
        torch.cuda.empty_cache()
        return s
    if kind == "hop":
        s["graph"] = synth.rmat_graph(case["nodes"], case["edges"], seed)
        g = torch.Generator("cuda").manual_seed(seed + 1)
        s["ids"] = torch.randint(case["nodes"], (case["rows"],), device="cuda", generator=g)
        s["seed"] = seed + 2
        return s
    s["graph"], renamed = _graph(case, seed)
    graph = s["graph"]
    store = _store(case["nodes"], case["dim"], case["dtype"], seed + 1)
    torch.cuda.empty_cache()
    options = dict(replace=case["replace"], weighted=case["weighted"], subgraph_type=case["subgraph"],
                   track_edge_ids=case["edge_ids"], seed=SAMPLER_SEED, rng_mode=case["rng"])
    fanout = _fanouts(case["fanout"])
    if kind == "epoch":
        split = renamed(np.random.default_rng(SEEDS_SEED).integers(0, case["nodes"], case["inputs"])).astype(np.int64)
        s["loader"] = EpochLoader(graph, fanout, input_nodes=split, batch_size=case["batch"], features=store,
                                  num_workers=case["threads"], prefetch_factor=case["depth"], group=case["group"], **options)
        return s
    cfg = ag.SamplingConfig(fanout, **options)
    s["seeds"] = [renamed(synth.seed_batch(case["nodes"], case["batch"], SEEDS_SEED, b)) for b in range(case["batches"])]
    if kind == "sample":
        s["sampler"] = ag.NeighborSampler(graph, cfg, features=store)
    else:
        s["loader"] = ag.NeighborLoader(graph, cfg, prefetch_depth=case["depth"], sampler_threads=case["threads"],
                                        features=store, group=case["group"])
    return s


# ---------------------------------------------------------------------- run --
def _batch(sg):
    return sg.x, sg.edge_index_local_t, sg.nodes_t, sg.edge_ids_t, sg.seed_indices_t


def _hetero_batch(sg):
    types = ("user", "post", "comment", "subreddit")
    return ([sg.nodes_t(t) for t in types], [sg.x_t(t) for t in types],
            [sg.edge_index_local_t(*r) for r in HETERO_RELATIONS], sg.seed_indices_t)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gather":
        return state["store"].gather(state["ids"])
    if kind == "get_batch":
        return state["store"].get_batch(state["ids"])
    if kind == "hop":
        return reservoir_hop(state["graph"], state["ids"], case["fanout"], state["seed"])
    if kind == "epoch":
        return [(b.x, b.edge_index, b.n_id, b.e_id, b.seed_index, b.input_id) for b in state["loader"]]
    if kind == "sample":
        return _batch(state["sampler"].sample(state["seeds"][0]))
    read = _hetero_batch if kind == "hetero" else _batch
    if "sampler" in state:
        return read(state["sampler"].sample("user", state["seeds"][0]))
    loader, out, asked = state["loader"], [], 0
    room = 4 * case["depth"]  # batches submitted ahead; the loader's own queue holds twice as many
    for _ in state["seeds"]:
        while asked < len(state["seeds"]) and asked - len(out) < room:
            loader.submit(asked, state["seeds"][asked])
            asked += 1
        out.append(read(loader.next_batch()[1]))
    return out


# --------------------------------------------------------------------- work --
# The size of a sampled subgraph is not in the case, so it is taken from a model of the
# graph: an R-MAT vertex's degree follows from the one bits of its id (a level is a source
# bit of 1 with probability 0.24), and the far end of its edges from the same bits (a bit
# is 1 with probability 0.05 / 0.24 or 0.19 / 0.76).  The model is walked once with a
# fixed random stream.  Single scattered reads cost a 32-byte sector.
def _bits(n):
    return max(1, (int(n) - 1).bit_length())


def _degrees(r, ids, n, edges):
    bits = _bits(n)
    ones = sum((ids >> b) & 1 for b in range(bits))
    return r.poisson(edges * 0.24 ** ones * 0.76 ** (bits - ones))


def _far_ends(r, ids, n_from, n_to):
    """One random edge's other end for every entry of ids; ends past n_to are drawn again."""
    bf, bt = _bits(n_from), _bits(n_to)
    out = np.zeros(len(ids), dtype=np.int64)
    todo = np.arange(len(ids))
    for _ in range(16):
        v, d = ids[todo], np.zeros(len(todo), dtype=np.int64)
        for b in range(bt):
            p = np.where((v >> b) & 1, 0.05 / 0.24, 0.25) if b < bf else 0.24
            d |= (r.random(len(todo)) < p).astype(np.int64) << b
        out[todo] = d % n_to
        todo = todo[d >= n_to]
        if not len(todo):
            break
    return out


def _sampled(case, seeds):
    """(nodes, edges, expanded vertices, row positions read in full, graph edges between the nodes) of one batch."""
    r = np.random.default_rng(7)
    n, e = case["nodes"], case["edges"]
    known = new = np.unique(r.integers(0, n, seeds))
    edges = expanded = scanned = 0
    for k in _fanouts(case["fanout"]):
        deg = _degrees(r, new, n, e)
        take = np.where(deg > 0, k, 0) if case["replace"] else np.minimum(deg, k)
        edges += int(take.sum())
        expanded += len(new)
        if case["weighted"]:
            scanned += int(deg[deg > k].sum())
        new = np.setdiff1d(_far_ends(r, np.repeat(new, take), n, n), known)
        known = np.union1d(known, new)
    between = 0.0
    if case["subgraph"] == "induced":
        deg = _degrees(r, known, n, e)
        scanned += int(deg.sum())
        probes = np.minimum(deg, 8)
        hit = np.isin(_far_ends(r, np.repeat(known, probes), n, n), known)
        between = float((hit * np.repeat(deg / np.maximum(probes, 1), probes)).sum())
    return len(known), edges, expanded, scanned, between


def _hetero_sampled(case):
    r = np.random.default_rng(7)
    sizes = _hetero_sizes(case["users"])
    total = {"votes": 30 * case["users"], "writes": 8 * case["users"], "belongs_to": sizes["post"]}
    fan = dict(zip(HETERO_RELATIONS, [_fanouts(f) for f in case["fanout"].split("/")] * 2))
    known = {t: np.zeros(0, dtype=np.int64) for t in sizes}
    known["user"] = np.unique(r.integers(0, sizes["user"], case["batch"]))
    new, edges, rows = dict(known), 0, 0
    for hop in range(2):
        found = {t: [np.zeros(0, dtype=np.int64)] for t in sizes}
        for (src, rel, dst), k in fan.items():
            ids, k = new[dst], k[hop]
            rows += len(ids)
            if "belongs_to" in rel:  # uniform: one subreddit per post, many posts per subreddit
                deg = np.full(len(ids), 1) if dst == "post" else r.poisson(sizes["post"] / sizes["subreddit"], len(ids))
            else:
                deg = _degrees(r, ids, sizes[dst], total[rel.removeprefix("rev_")])
            take = np.where(deg > 0, k, 0) if case["replace"] else np.minimum(deg, k)
            at = np.repeat(ids, take)
            edges += len(at)
            found[src].append(r.integers(0, sizes[src], len(at)) if "belongs_to" in rel else _far_ends(r, at, sizes[dst], sizes[src]))
        new = {t: np.setdiff1d(np.concatenate(f), known[t]) for t, f in found.items()}
        known = {t: np.union1d(known[t], new[t]) for t in sizes}
    return {t: len(v) for t, v in known.items()}, edges, rows


def _row_bytes(case, dim=None):
    """One stored row read (whole sectors, int8 with its scales) and its f32 decode written."""
    dim = dim or case["dim"]
    stored = dim * ELEMENT[case["dtype"]]
    scales = -(-dim // 32) * 4 if case["dtype"] == "i8" else 0
    return -(-stored // 32) * 32 + scales + 4 * dim


def work(case):
    kind = case["kind"]
    if kind in ("gather", "get_batch"):
        return {"bytes": case["rows"] * (8 + _row_bytes(case)), "flops": 0}
    if kind == "hop":
        r = np.random.default_rng(7)
        k = case["fanout"]
        deg = _degrees(r, r.integers(0, case["nodes"], case["rows"]), case["nodes"], case["edges"])
        picks = np.minimum(deg, k) if k <= 32 else np.where(deg > 0, k, 0)
        return {"bytes": case["rows"] * (8 + 32 + 4 + 4 * k) + 32 * int(picks.sum()), "flops": 0}
    if kind == "hetero":
        nodes, edges, rows = _hetero_sampled(case)
        # a row's bounds and a source per edge, then ids, edge_index and feature rows
        one = 32 * rows + edges * (32 + 16) + sum(n * (8 + _row_bytes(case, 64 if t == "subreddit" else None)) for t, n in nodes.items())
        return {"bytes": case["batches"] * one, "flops": 0}
    batches = case["batches"] if kind != "epoch" else case["inputs"] / case["batch"]
    nodes, edges, expanded, scanned, between = _sampled(case, case["batch"])
    # per expanded vertex its row bounds, per edge a destination; scanned positions 4 bytes each
    kept = between if case["subgraph"] == "induced" else edges
    one = 32 * expanded + 32 * edges + 4 * scanned + kept * (16 + 8 * case["edge_ids"]) + nodes * (8 + _row_bytes(case)) + 12 * case["batch"]
    return {"bytes": int(batches * one), "flops": 0}


def tolerance(case):
    # Ids, positions and exact decodes of stored values: the sampler reproduces a defined
    # random stream bit for bit, and f16 / bf16 / int8 decode without rounding freedom.
    return "exact"
