"""Batches at the edges of the sampling kernels' tiles: seed counts around one tile of every
size, and stages large enough for each number of items per thread, against the CPU oracle."""
import numpy as np
import pytest

from helpers import assert_same_subgraph, csr_from_edges

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    import aethergraph_b200 as ag

    rng = np.random.default_rng(8)
    n, e = 300_000, 2_400_000
    off, dst, _ = csr_from_edges(n, rng.integers(0, n, e).astype(np.uint32), rng.integers(0, n, e).astype(np.uint32))
    return n, off, dst, ag.Graph.from_csr(off, dst)


@pytest.mark.parametrize("n_seeds", [1, 511, 512, 513, 1024, 1025, 2048, 2049, 160_000, 320_000, 400_000])
def test_seed_counts(graph, n_seeds):
    import aethergraph_b200 as ag
    from oracle import ago

    n, off, dst, g = graph
    rng = np.random.default_rng(n_seeds)
    s = ag.NeighborSampler(g, ag.SamplingConfig(num_neighbors=[2, 1], seed=5))
    o = ago.Sampler(off, dst, [2, 1], seed=5)
    for _ in range(2):  # sized from the bounds, then from the first batch's counts
        seeds = rng.integers(0, n, n_seeds).astype(np.uint32)
        assert_same_subgraph(s.sample(seeds).raw_u32(), o.sample(seeds))


@pytest.mark.parametrize("n_seeds", [700, 2100, 30_000])
def test_groups(graph, n_seeds):
    import aethergraph_b200 as ag
    from oracle import ago

    n, off, dst, g = graph
    rng = np.random.default_rng(n_seeds)
    batches = [rng.integers(0, n, n_seeds - 13 * i).astype(np.uint32) for i in range(8)]
    o = ago.Sampler(off, dst, [3, 2], seed=5)
    got = ag.ParallelBatchSampler(g, ag.SamplingConfig(num_neighbors=[3, 2], seed=5), streams=2, group=4).sample_batches(batches)
    for i, (sg, b) in enumerate(zip(got, batches)):
        o.reseed(ago.batch_seed(5, i))
        assert_same_subgraph(sg.raw_u32(), o.sample(b), ctx=f"batch {i}: ")
