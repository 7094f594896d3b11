"""Heterogeneous chains at the edges of their launch forms, against the CPU oracle: the staged
block in kernel parameters of every size or copied, class ranks over more tiles than one
look-back window, and the node types' rows gathered together or type by type."""
import numpy as np
import pytest

from helpers import csr_from_edges
from test_hetero_gpu import _same

pytestmark = pytest.mark.gpu

N = {"a": 60_000, "b": 40_000}
ETS = [("a", "to", "b"), ("b", "back", "a"), ("a", "self", "a")]
FAN = [[6, 3], [32, 4], [5, 2]]


@pytest.fixture(scope="module")
def graph():
    import aethergraph_b200 as ag

    rng = np.random.default_rng(2)
    names, edges, rels = list(N), [], []
    for s, _, d in ETS:
        e = 20 * N[s]
        edges.append((rng.integers(0, N[s], e).astype(np.uint32), rng.integers(0, N[d], e).astype(np.uint32)))
        off, dst, _ = csr_from_edges(N[s], *edges[-1])
        rels.append((names.index(s), names.index(d), off, dst))
    return ag.HeteroCsrGraph.from_edge_arrays(N, [(*et, *e) for et, e in zip(ETS, edges)]), rels


def _stores(dims, dtypes):
    import aethergraph_b200 as ag

    rng = np.random.default_rng(5)
    return {t: ag.FeatureStore.from_array(rng.standard_normal((N[t], d)).astype(np.float32), dtype=k) for t, d, k in zip(N, dims, dtypes)}


@pytest.mark.parametrize("n_seeds", [1, 700, 1500, 3500, 5000])
def test_seed_counts(graph, n_seeds):
    import aethergraph_b200 as ag
    from oracle import ago

    g, rels = graph
    s = ag.HeteroNeighborSampler(g, ag.HeteroSamplingConfig(dict(zip(ETS, FAN)), seed=8))
    o = ago.HeteroSampler(list(N.values()), rels, FAN, seed=8)
    for i in range(2):  # sized from the bounds, then from the first batch's counts
        seeds = np.random.default_rng(n_seeds + i).integers(0, N["a"], n_seeds).astype(np.uint32)
        _same(s.sample("a", seeds).raw_u32(), o.sample(0, seeds))


@pytest.mark.parametrize("dims,dtypes", [((64, 256), ("bf16", "bf16")), ((8, 136), ("f16", "f16")), ((64, 64), ("f32", "bf16")),
                                         ((64, 33), ("f16", "f16")), ((64, 128), ("i8", "i8"))])
@pytest.mark.parametrize("group", [1, 4])
def test_rows_of_every_type(graph, dims, dtypes, group):
    import torch

    import aethergraph_b200 as ag
    from oracle import ago

    g, rels = graph
    stores = _stores(dims, dtypes)
    batches = [np.random.default_rng(i).integers(0, N["a"], 300 + i).astype(np.uint32) for i in range(6)]
    ld = ag.HeteroNeighborLoader(g, ag.HeteroSamplingConfig(dict(zip(ETS, FAN)), seed=8), "a", prefetch_depth=4, features=stores,
                                 sampler_threads=2, group=group)
    o = ago.HeteroSampler(list(N.values()), rels, FAN, seed=8)
    for i, b in enumerate(batches):
        ld.submit(i, b)
    for i, b in enumerate(batches):
        _, sg = ld.next_batch()[:2]
        o.reseed(ago.batch_seed(8, i))
        _same(sg.raw_u32(), o.sample(0, b))
        for t in N:
            assert torch.equal(sg.x_t(t), stores[t].gather(sg.nodes_t(t)))
    ld.shutdown()
