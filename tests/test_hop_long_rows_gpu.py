"""One-hop Philox sampling of rows around the lengths where a warp takes over from a decision per
lane and a block from a warp, in launches of one and of four rows per warp,
against the CPU oracle."""
import numpy as np
import pytest

from helpers import csr_from_edges

pytestmark = pytest.mark.gpu

DEGREES = [2047, 2048, 2049, 5, 33, 34, 6, 100_003, 7, 0, 1, 2, 4, 3000, 37, 38, 39, 40, 64, 65]


@pytest.mark.parametrize("fanout", [1, 5, 6, 7, 32, 40])
@pytest.mark.parametrize("copies", [1, 900, 1500])
def test_long_rows(fanout, copies):
    import aethergraph_b200 as ag
    from aethergraph_b200.sampler import reservoir_hop
    from oracle import ago

    n = len(DEGREES)
    rng = np.random.default_rng(1)
    src = np.repeat(np.arange(n), DEGREES).astype(np.uint32)
    off, dst, _ = csr_from_edges(n, src, rng.integers(0, n, len(src)).astype(np.uint32))
    g = ag.Graph.from_csr(off, dst)
    nodes = np.concatenate([np.tile(np.arange(n)[::-1], copies), [n, n + 5]])  # two outside the graph
    out, counts = reservoir_hop(g, nodes, fanout, 99, 1)
    out, counts = out.cpu().numpy().view(np.uint32), counts.cpu().numpy()
    want = {}
    for v in range(n):
        row = dst[int(off[v]):int(off[v + 1])]
        if fanout > 32 and len(row):
            want[v] = np.array([row[ago.philox_u32(99, 1, v, d) % len(row)] for d in range(fanout)], dtype=np.uint32)
        else:
            want[v] = ago.reservoir_sample(row, fanout, 99, 1, v) if len(row) else row
    for i, v in enumerate(nodes):
        w = want.get(int(v), np.zeros(0, dtype=np.uint32))
        assert counts[i] == len(w) and np.array_equal(out[i, :len(w)], w) and (out[i, len(w):] == 0xFFFFFFFF).all()
