"""Rows that are not whole 16-byte vectors, and outputs that are not 16-byte aligned, bit for
bit against a plain decode: every unit size, every number of lanes per row, ragged counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _decoded(store, n, dim, dtype):
    raw = store.payload_to_host().reshape(n, dim)
    if dtype == "f32":
        return raw
    if dtype == "bf16":
        return (raw.astype(np.uint32) << 16).view(np.float32)
    if dtype == "f16":
        return raw.view(np.float16).astype(np.float32)
    scales = np.repeat(store.scales_to_host(), 32, axis=1)[:, :dim]
    return raw.astype(np.float32) * scales


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16", "i8"])
@pytest.mark.parametrize("dim", [1, 2, 5, 6, 7, 9, 20, 33, 50, 63, 100, 130, 301, 602])
def test_rows_and_offsets(dtype, dim):
    import torch

    import aethergraph_b200 as ag

    n = 500
    rng = np.random.default_rng(dim)
    x = (rng.standard_normal((n, dim)) * 10.0 ** rng.integers(-4, 3, (n, 1))).astype(np.float32)
    store = ag.FeatureStore.from_array(x, dtype)
    want = _decoded(store, n, dim, dtype)
    for rows, shift, kind in ((1, 0, torch.int64), (777, 0, torch.int32), (777, 1, torch.int64), (300, 2, torch.int32)):
        ids = rng.integers(0, n, rows)
        buf = torch.full((rows * dim + 8,), 7.0, device="cuda")
        out = buf[shift:shift + rows * dim].view(rows, dim)
        store.gather(torch.from_numpy(ids).to("cuda", dtype=kind), out=out)
        got = buf.cpu().numpy()
        assert np.array_equal(got[shift:shift + rows * dim].reshape(rows, dim).view(np.uint32), want[ids].view(np.uint32))
        assert (got[:shift] == 7).all() and (got[shift + rows * dim:] == 7).all()


@pytest.mark.parametrize("dtype,dim,rows", [
    ("f32", 5, 30_000), ("f32", 5, 70_001), ("f32", 1, 400_003), ("bf16", 6, 200_001), ("i8", 9, 50_000),  # short rows: few units, many
    ("f16", 100, 7000), ("f16", 100, 9001), ("f32", 25, 20_011), ("i8", 128 - 4, 13_001),                   # one step of a lane group
    ("f32", 17, 30_011), ("bf16", 33, 20_003), ("i8", 301, 1999), ("f16", 602, 3001),                       # row by row
    ("f32", 4099, 1), ("f32", 4099, 101), ("f16", 4099, 300), ("i8", 1023, 777), ("bf16", 8190, 40),        # steps on blocks of their own
])
def test_launch_forms(dtype, dim, rows):
    """Few units, short rows, row by row, rows in steps: every element, and ids outside the store."""
    import torch

    import aethergraph_b200 as ag

    n = 300
    rng = np.random.default_rng(rows)
    store = ag.FeatureStore.from_array(rng.standard_normal((n, dim)).astype(np.float32), dtype)
    ids = rng.integers(0, n, rows)
    want = torch.from_numpy(_decoded(store, n, dim, dtype)).cuda()[torch.from_numpy(ids).cuda()]
    assert torch.equal(store.gather(torch.from_numpy(ids).cuda()).view(torch.int32), want.view(torch.int32))
    store.check()
    bad = np.unique(rng.integers(0, rows, 5))
    ids[bad] = n + bad
    want[torch.from_numpy(bad).cuda()] = 0
    assert torch.equal(store.gather(torch.from_numpy(ids).cuda()).view(torch.int32), want.view(torch.int32))
    with pytest.raises(ValueError):
        store.check()


@pytest.mark.parametrize("dtype,dim,rows", [("f32", 5, 1000), ("bf16", 5, 70_001), ("f16", 100, 9001), ("f16", 33, 20_003), ("f32", 4099, 101)])
def test_launch_forms_of_a_sharded_view(dtype, dim, rows):
    import torch

    import aethergraph_b200 as ag
    from aethergraph_b200 import synth

    n, world = 301, 3
    whole = synth.features(n, dim, dtype, 7)
    ids = torch.from_numpy(np.random.default_rng(rows).integers(0, n, rows)).cuda()
    want = torch.from_numpy(_decoded(whole, n, dim, dtype)).cuda()[ids]
    for layout in ("range", "cyclic"):
        shards = [synth.features_shard(n, dim, dtype, 7, r, world, layout) for r in range(world)]
        view = ag.FeatureStore.view_sharded(shards, 1)
        assert torch.equal(view.gather(ids).view(torch.int32), want.view(torch.int32))
        view.check()


@pytest.mark.parametrize("dtype,dim", [("f16", 100), ("bf16", 301), ("f32", 50), ("i8", 100)])
def test_batches_of_a_chain(dtype, dim):
    import torch

    import aethergraph_b200 as ag
    from helpers import rmat_csr

    n, off, dst, _ = rmat_csr(11, 8, seed=3)
    x = np.random.default_rng(1).standard_normal((n, dim)).astype(np.float32)
    store = ag.FeatureStore.from_array(x, dtype)
    want = _decoded(store, n, dim, dtype)
    batches = [np.random.default_rng(i).integers(0, n, 90 + i).astype(np.uint32) for i in range(5)]
    sampler = ag.ParallelBatchSampler(ag.Graph.from_csr(off, dst), ag.SamplingConfig(num_neighbors=[5, 3], seed=2), features=store, group=4)
    for sg in sampler.sample_batches(batches):
        assert torch.equal(sg.x.cpu(), torch.from_numpy(want[sg.nodes]))


def test_bad_ids_decode_to_zeros_and_are_reported():
    import torch

    import aethergraph_b200 as ag

    store = ag.FeatureStore.from_array(np.ones((10, 50), dtype=np.float32), "f16")
    out = store.gather(torch.tensor([3, 10, 4], device="cuda"))
    assert out[0].eq(1).all() and out[1].eq(0).all() and out[2].eq(1).all()
    with pytest.raises(ValueError):
        store.check()


@pytest.mark.parametrize("dim", [1, 256])
def test_every_f16_pattern(dim):
    import aethergraph_b200 as ag
    from oracle import ago

    bits = np.arange(65536, dtype=np.uint16).reshape(-1, dim)
    store = ag.FeatureStore.from_payload(bits, 65536 // dim, dim, "f16")
    assert np.array_equal(store.features().view(np.uint32), ago.decode(bits, "f16").reshape(-1, dim).view(np.uint32))
