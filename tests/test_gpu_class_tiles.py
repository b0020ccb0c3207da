"""Unique + relabel by classes of ids in tiles that sort themselves, against the oracle: minibatches that end at, before and behind a
tile, empty ones among them, runs longer than a warp keeps, more tiles than a warp knows, ids that crowd, lie beyond the bound or are
no ids.  The automatic choice on both sides of its bound."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TILE = 16_384


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def tiles():
    from graph_sampling_b200 import ops
    ctx = ops.Context()
    ctx.set_option("relabel_path", 5)
    return ctx


def ids(rng, count, nodes, kind):
    if kind == "fourth":
        return (nodes * rng.random(count) ** 4).astype(np.int64)
    if kind == "one":
        return np.full(count, nodes // 3)
    if kind == "even":
        return rng.integers(0, nodes, count)
    step = int(kind)
    return step * rng.integers(0, (nodes - 1) // step + 1, count)


def check(oracle, got, seeds, sp, edges, ep):
    uniq, up, rel = (t.cpu().numpy() for t in got[:3])
    assert up[0] == 0 and up[-1] == len(uniq) and len(rel) == ep[-1]
    for b in range(len(sp) - 1):
        e = edges[ep[b]:ep[b + 1]]
        want, (w_rel,) = oracle.unique_relabel([seeds[sp[b]:sp[b + 1]], e], [e])
        np.testing.assert_array_equal(uniq[up[b]:up[b + 1]], want)
        np.testing.assert_array_equal(rel[ep[b]:ep[b + 1]], w_rel)


def call(seeds, sp, edges, ep, nodes, ctx):
    from graph_sampling_b200 import ops
    return ops.batch_csr_relabel(dev(seeds), dev(sp), dev(edges), dev(ep), num_nodes=nodes, ctx=ctx)


@pytest.mark.parametrize("kind", ["even", "fourth", "one", "11", "13", "151"])
@pytest.mark.parametrize("nodes", [900, 180_225, 2_450_000, 4_177_920])
def test_minibatches_around_a_tile(oracle, nodes, kind):
    rng = np.random.default_rng(nodes)
    items = np.array([0, 1, TILE - 1, TILE, 0, TILE + 1, 3 * TILE, 0, 5 * TILE + 77, 0])
    ns = items // 5
    sp, ep = np.concatenate([[0], np.cumsum(ns)]), np.concatenate([[0], np.cumsum(items - ns)])
    seeds, edges = ids(rng, sp[-1], nodes, "even"), ids(rng, ep[-1], nodes, kind)
    check(oracle, call(seeds, sp, edges, ep, nodes, tiles()), seeds, sp, edges, ep)


def test_more_tiles_than_a_warp_knows(oracle):
    rng = np.random.default_rng(1)
    sp, ep = np.array([0, 100, 100, 1100]), np.array([0, 50_000, 50_000, 50_000 + 530 * TILE])   # 32 runs of a warp, and 530 of all
    seeds, edges = ids(rng, sp[-1], 2_450_000, "even"), ids(rng, ep[-1], 2_450_000, "fourth")
    check(oracle, call(seeds, sp, edges, ep, 2_450_000, tiles()), seeds, sp, edges, ep)


def test_ids_beyond_the_bound_and_no_ids(oracle):
    from graph_sampling_b200.cabi import GsbError
    rng = np.random.default_rng(2)
    sp, ep, nodes = np.array([0, 3000, 6000]), np.array([0, 40_000, 120_000]), 200_000
    seeds, edges = ids(rng, sp[-1], nodes, "even"), ids(rng, ep[-1], nodes, "fourth")
    edges[::3] = 2**32 - 2 - ids(rng, len(edges[::3]), 5000, "even")
    seeds[::7] = 300_000 + ids(rng, len(seeds[::7]), 1000, "even")
    check(oracle, call(seeds, sp, edges, ep, nodes, tiles()), seeds, sp, edges, ep)
    for bad in (-1, 2**32 - 1, 2**40):
        wrong = edges.copy()
        wrong[50_000] = bad
        ctx = tiles()
        with pytest.raises(GsbError) as e:
            call(seeds, sp, wrong, ep, nodes, ctx)
        assert e.value.status == -8
        check(oracle, call(seeds, sp, edges, ep, nodes, ctx), seeds, sp, edges, ep)


def test_batched_unique_and_hops(oracle):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(3)
    degree = rng.integers(0, 40, 30_000)
    indptr = np.concatenate([[0], np.cumsum(degree)])
    indices = rng.integers(0, 30_000, indptr[-1])
    seeds, ptr = rng.integers(0, 30_000, 9000), np.array([0, 4000, 4000, 9000])
    hops = [ops.sage_sample_batches(dev(indptr), dev(indices), dev(seeds), dev(ptr), [10, 5], seed=3, ctx=ctx)
            for ctx in (tiles(), ops.Context())]
    for a, b in zip(*hops):
        for key in a:
            assert torch.equal(a[key], b[key]), key


# 2 450 000 nodes are 151 classes: 106 400 items a minibatch
@pytest.mark.parametrize("items", [106_399, 106_400])
def test_automatic_choice(oracle, items):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(items)
    G, nodes, ns = 12, 2_450_000, items // 6
    sp, ep = np.arange(G + 1) * ns, np.arange(G + 1) * (items - ns)
    seeds, edges = ids(rng, sp[-1], nodes, "even"), ids(rng, ep[-1], nodes, "fourth")
    check(oracle, call(seeds, sp, edges, ep, nodes, ops.Context()), seeds, sp, edges, ep)
