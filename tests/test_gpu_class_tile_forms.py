"""Class tiles and sampling by windows where their tests don't go: runs cut into pieces and more pieces than a warp keeps, the last
number of tiles whose positions fit a table word and the first that don't, which calls take the form, waits that run out in their
look-backs, bounds that are too small."""
import numpy as np
import pytest
import torch

from tests.test_gpu_bounded_waits import dev, graph, pinned, run_out

pytestmark = pytest.mark.gpu
TILE = 16_384


@pytest.fixture(scope="module")
def ops():
    from graph_sampling_b200 import ops as _ops
    return _ops


def relabel(ops, seeds, sp, edges, ep, nodes, path):
    ctx = ops.Context()
    ctx.set_option("relabel_path", path)
    got = ops.batch_csr_relabel(dev(seeds), dev(sp), dev(edges), dev(ep), num_nodes=nodes, ctx=ctx)[:3]
    return [t.cpu().numpy() for t in got], ctx.launch_count()


# 180 000 nodes are 11 classes, whose runs of 1 500 words are cut into eight pieces: 16 warps keep four of them each up to eight tiles
@pytest.mark.parametrize("nodes,tiles", [(180_000, (8, 9, 17)), (180_000, (63, 1, 64)), (700_000, (50, 3)), (1_000_000, (63, 64))])
def test_pieces_of_runs_and_positions(oracle, ops, nodes, tiles):
    rng = np.random.default_rng(nodes + len(tiles))
    items = np.array(tiles) * TILE
    ns = items // 7
    sp, ep = np.concatenate([[0], np.cumsum(ns)]), np.concatenate([[0], np.cumsum(items - ns)])
    seeds, edges = rng.integers(0, nodes, sp[-1]), (nodes * rng.random(ep[-1]) ** 3).astype(np.int64)
    (uniq, up, rel), _ = relabel(ops, seeds, sp, edges, ep, nodes, 5)
    assert up[0] == 0 and up[-1] == len(uniq) and len(rel) == ep[-1]
    for b in range(len(tiles)):
        e = edges[ep[b]:ep[b + 1]]
        want, (w_rel,) = oracle.unique_relabel([seeds[sp[b]:sp[b + 1]], e], [e])
        np.testing.assert_array_equal(uniq[up[b]:up[b + 1]], want)
        np.testing.assert_array_equal(rel[ep[b]:ep[b + 1]], w_rel)


# six launches in tiles, eight in buckets
@pytest.mark.parametrize("nodes,G,items,tiled", [(2_450_000, 12, 106_399, False), (2_450_000, 12, 106_400, True),
                                                 (2_450_000, 12, 243_300, False), (700_000, 112, 35_999, False),
                                                 (700_000, 112, 36_000, True), (500_000, 112, 36_000, False)])
def test_which_calls_take_tiles(ops, nodes, G, items, tiled):
    rng = np.random.default_rng(items)
    ns = items // 6
    sp, ep = np.arange(G + 1) * ns, np.arange(G + 1) * (items - ns)
    seeds, edges = rng.integers(0, nodes, sp[-1]), (nodes * rng.random(ep[-1]) ** 4).astype(np.int64)
    got, launches = relabel(ops, seeds, sp, edges, ep, nodes, 0)
    assert launches == (6 if tiled else 8)
    want, launches = relabel(ops, seeds, sp, edges, ep, nodes, 3)
    assert launches == 8 and all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("k", [5, 16])
def test_waits_in_windows(ops, k):
    indptr, indices = graph(100_000, 2_000_000, 6)
    columns = pinned(np.random.default_rng(k).integers(0, 100_000, 300_000))

    def call(ctx):
        ctx.set_option("sample_path", 2)
        return ops.fused_csc_col_slicing_sampling(indptr, indices, columns, k, False, seed=3, ctx=ctx)

    run_out(ops, call)


def test_waits_in_tiles(ops):
    rng = np.random.default_rng(7)
    sp, ep = np.arange(41) * 500, np.arange(41) * 12_000
    seeds, edges = dev(rng.integers(0, 50_000, sp[-1])), dev(rng.integers(0, 50_000, ep[-1]))
    d_sp, d_ep = dev(sp), dev(ep)

    def call(ctx):
        ctx.set_option("relabel_path", 5)
        return ops.batch_csr_relabel(seeds, d_sp, edges, d_ep, ctx=ctx, num_nodes=50_000)[:3]

    run_out(ops, call, tries=50, certain=False)


@pytest.mark.parametrize("relabel_path,sample_path", [(5, 0), (5, 2), (3, 2), (4, 2), (1, 2)])
def test_waits_in_queued_hops(ops, relabel_path, sample_path):
    indptr, indices = graph(100_000, 2_000_000, 5)
    seeds, ptr = pinned(np.arange(16_000)), dev(np.arange(17) * 1000)

    def call(ctx):
        ctx.set_option("relabel_path", relabel_path)
        ctx.set_option("sample_path", sample_path)
        hops = ops.sage_sample_batches(indptr, indices, seeds, ptr, [5, 5, 3], seed=2, ctx=ctx, sync=False)
        return [h["frontier_ptr"] for h in hops]

    run_out(ops, call)


@pytest.mark.parametrize("sample_path", [1, 2])
def test_too_small_a_bound_in_tiles(ops, sample_path):
    from graph_sampling_b200.cabi import GsbError
    indptr, indices = graph(100_000, 2_000_000, 5)
    ctx = ops.Context()
    ctx.set_option("relabel_path", 5)
    ctx.set_option("sample_path", sample_path)
    args = (indptr, indices, dev(np.arange(16_000)), dev(np.arange(5) * 4000), [5, 3])
    edges = int(torch.diff(indptr[:16_001]).clamp(max=5).sum())
    ops.sage_sample_batches(*args, seed=1, ctx=ctx, sync=False, size_hints=[(16_000, edges - 1), (50_000, 100_000)])
    with pytest.raises(GsbError) as e:
        ctx.check_device()
    assert e.value.status == -4
    for a, b in zip(ops.sage_sample_batches(*args, seed=1, ctx=ctx), ops.sage_sample_batches(*args, seed=1)):
        for key in a:
            assert torch.equal(a[key], b[key]), key
