"""Rows far longer than the rest of their hop, against the CPU oracle, at the edges of the
slices they are split into."""
import numpy as np
import pytest

from helpers import assert_same_subgraph, csr_from_edges

pytestmark = pytest.mark.gpu


def _hub_graph(degrees, n, seed, weights=None):
    """Vertex i < len(degrees) has degrees[i] neighbours, every other vertex five of them hubs."""
    rng = np.random.default_rng(seed)
    src = [np.full(d, i) for i, d in enumerate(degrees)] + [np.repeat(np.arange(len(degrees), n), 5)]
    src = np.concatenate(src).astype(np.uint32)
    dst = rng.integers(0, n, len(src)).astype(np.uint32)
    low = src >= len(degrees)
    dst[low] = rng.integers(0, len(degrees), int(low.sum()))
    w = None
    if weights == "lognormal":
        w = rng.lognormal(0.0, 1.0, len(src)).astype(np.float32)
    elif weights == "equal":
        w = np.ones(len(src), dtype=np.float32)
    elif weights == "odd":  # zeros, negatives, infinities, NaN and subnormal weights never win before a real one
        w = rng.lognormal(0.0, 1.0, len(src)).astype(np.float32)
        w[rng.random(len(w)) < 0.9995] = 0.0
        for value in (-1.0, np.inf, np.nan, 1e-42, 3.3e38, 1e-30):
            w[rng.integers(0, len(w), 50)] = value
    elif weights == "pareto":  # no mean: the sampled weights say little about the keys
        w = (1.0 + rng.pareto(0.5, len(src))).astype(np.float32)
    elif weights in ("heavy", "few"):  # a row's first position far above the rest; eight positive ones and zeros
        at = np.arange(len(src)) - np.searchsorted(src, src)
        w = np.where(at == 0, 1e6, 1.0) if weights == "heavy" else np.where(at % 61 == 0, 1.0, 0.0) * (at < 8 * 61)
        w = w.astype(np.float32)
    elif weights == "comb":  # positive exactly where a row's mean weight is sampled
        at = np.arange(len(src)) - np.searchsorted(src, src)
        w = (at % np.maximum(np.bincount(src)[src] // 512, 1) == 0).astype(np.float32)
    return csr_from_edges(n, src, dst, w)


DEGREES = [2047, 2048, 2049, 4096, 4097, 31, 33, 70_000, 530_001, 9000, 0, 1, 16, 15]
# and at the edges of a chunk, of the rows that start from a guessed threshold and of its sample
WEIGHTED_DEGREES = DEGREES + [32, 64, 65, 127, 128, 129, 160, 511, 512, 513, 1500]


@pytest.mark.parametrize("weights", ["lognormal", "equal", "odd", "pareto", "heavy", "few", "comb"])
@pytest.mark.parametrize("fanout", [[15, 4], [32], [1, 1, 2]])
def test_weighted(weights, fanout):
    """With "heavy", "few" and "comb" the guessed threshold is below the k-th best key of most long
    rows, with "comb" of those above 1024 that stay with a warp too: they are streamed once more."""
    import aethergraph_b200 as ag
    from oracle import ago

    n = 4000
    off, dst, w = _hub_graph(WEIGHTED_DEGREES, n, 3, weights)
    g = ag.Graph.from_csr(off, dst, w)
    cfg = ag.SamplingConfig(num_neighbors=fanout, weighted=True, seed=11)
    o = ago.Sampler(off, dst, fanout, weights=w, weighted=True, seed=11)
    s = ag.NeighborSampler(g, cfg)
    for count in (len(WEIGHTED_DEGREES), 1, 60):
        seeds = np.arange(count, dtype=np.uint32)[::-1].copy()
        assert_same_subgraph(s.sample(seeds).raw_u32(), o.sample(seeds))
    batches = [np.arange(len(WEIGHTED_DEGREES) - i, dtype=np.uint32) for i in range(8)]
    for i, sg in enumerate(ag.ParallelBatchSampler(g, cfg, group=8).sample_batches(batches)):
        o.reseed(ago.batch_seed(11, i))
        assert_same_subgraph(sg.raw_u32(), o.sample(batches[i]), ctx=f"batch {i}: ")


def _philox(seed, layer, node, groups):
    """Philox4x32-10 blocks (node, layer, group), the generator's definition in numpy."""
    c = [np.full(len(groups), node & 0xFFFFFFFF, dtype=np.uint64), np.full(len(groups), node >> 32, dtype=np.uint64),
         np.full(len(groups), layer, dtype=np.uint64), groups.astype(np.uint64)]
    k0, k1, low = seed & 0xFFFFFFFF, seed >> 32, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return np.stack(c, axis=1)


@pytest.mark.parametrize("weights", ["lognormal", "few"])
@pytest.mark.parametrize("k", [1, 15, 32])
def test_weighted_philox(weights, k):
    """The counter-based stream has a filter of its own: position i draws words 2 i (high) and
    2 i + 1 of its vertex; the k smallest (key, position) win."""
    import aethergraph_b200 as ag
    from oracle import ago

    seed = 2**40 + 77
    assert list(_philox(seed, 1, 5, np.array([3]))[0]) == [ago.philox_u32(seed, 1, 5, 12 + i) for i in range(4)]
    degrees = [127, 128, 129, 2047, 2048, 2049, 4097, 70_000, 33, 64]
    off, dst, w = _hub_graph(degrees, 2000, 3, weights)
    want = {}
    for v, d in enumerate(degrees):
        words = _philox(seed, 0, v, np.arange((2 * d + 3) // 4)).reshape(-1)
        u = (((words[0:2 * d:2] << np.uint64(32)) | words[1:2 * d:2]) >> np.uint64(11)).astype(np.float64) + 1.0
        row = w[int(off[v]):int(off[v]) + d].astype(np.float64)
        with np.errstate(divide="ignore"):
            key = np.where(row > 0, -np.log(u / 2.0**53) / row, np.inf)
        want[v] = int(off[v]) + np.lexsort((np.arange(d), key))[:k]
    g = ag.Graph.from_csr(off, dst, w)
    cfg = ag.SamplingConfig(num_neighbors=[k], weighted=True, seed=seed, rng_mode="philox")
    seeds = np.arange(len(degrees), dtype=np.uint32)

    def check(raw):
        assert np.array_equal(raw["edge_src"], np.repeat(seeds, [min(k, d) for d in degrees]))
        assert np.array_equal(raw["edge_ids"].astype(np.int64), np.concatenate([want[v] for v in seeds]))

    check(ag.NeighborSampler(g, cfg).sample(seeds).raw_u32())


@pytest.mark.parametrize("rows,length,weights", [
    (1100, 2100, "lognormal"),  # rows that do not fit stay with their own warp
    (40, 66_000, "few"),        # these do fit, but not the shorter slices of rows whose guess was too low
])
def test_more_slices_than_the_queue_holds(rows, length, weights):
    import aethergraph_b200 as ag
    from oracle import ago

    group, queue = 64, 65_536
    first, again = -(-length // (16 * 2048)), -(-length // 2048)  # slices of a row: first launch of a chain this long, second
    assert group * rows * (again if weights == "few" else first) > queue
    assert weights != "few" or group * rows * first <= queue
    off, dst, w = _hub_graph([length] * rows, 2000, 5, weights)
    g = ag.Graph.from_csr(off, dst, w)
    cfg = ag.SamplingConfig(num_neighbors=[10], weighted=True, seed=4)
    o = ago.Sampler(off, dst, [10], weights=w, weighted=True, seed=4)
    batches = [np.roll(np.arange(rows, dtype=np.uint32), i) for i in range(group)]
    for i, sg in enumerate(ag.ParallelBatchSampler(g, cfg, streams=1, group=group).sample_batches(batches)):
        if i % 8 and i < group - 3:
            continue  # the restatement takes its time
        o.reseed(ago.batch_seed(4, i))
        assert_same_subgraph(sg.raw_u32(), o.sample(batches[i]), ctx=f"batch {i}: ")


@pytest.mark.parametrize("track", [True, False])
@pytest.mark.parametrize("degrees,seeds", [(DEGREES, 14), ([700_000], 1), ([0, 0, 0], 3), ([127, 128, 129, 160], 200), ([3] * 50, 0)])
def test_induced(degrees, seeds, track):
    import aethergraph_b200 as ag
    from oracle import ago

    n = 4000
    off, dst, _ = _hub_graph(degrees, n, 7)
    g = ag.Graph.from_csr(off, dst)
    s = ag.NeighborSampler(g, ag.SamplingConfig(num_neighbors=[6, 4], subgraph_type="induced", seed=2, track_edge_ids=track))
    o = ago.Sampler(off, dst, [6, 4], seed=2, track_edge_ids=track)
    for ids in (np.arange(seeds), np.arange(seeds)[::-1] * 7 % n):
        ids = ids.astype(np.uint32)
        sg, want = s.sample(ids), ago.induce(off, dst, o.sample(ids))
        assert_same_subgraph(sg.raw_u32(), want)
        eil = sg.edge_index_local
        assert np.array_equal(eil[0], want["dst_local"].astype(np.int64)) and np.array_equal(eil[1], want["src_local"].astype(np.int64))


def test_induced_without_the_node_filter():
    """More sampled nodes than the walk keeps a filter for."""
    import aethergraph_b200 as ag
    from oracle import ago

    rng = np.random.default_rng(9)
    n = 200_000
    off, dst, _ = csr_from_edges(n, rng.integers(0, n, 3 * n).astype(np.uint32), rng.integers(0, n, 3 * n).astype(np.uint32))
    seeds = rng.permutation(n)[:140_000].astype(np.uint32)
    s = ag.NeighborSampler(ag.Graph.from_csr(off, dst), ag.SamplingConfig(num_neighbors=[1], subgraph_type="induced", seed=2))
    assert_same_subgraph(s.sample(seeds).raw_u32(), ago.induce(off, dst, ago.Sampler(off, dst, [1], seed=2).sample(seeds)))
