"""The partitioned unique + relabel with buckets that are classes of up to 16 384 ids: few classes and many, ids at multiples of
16 384 and on both sides of the bound (those beyond it take a bucket of their own), buckets larger than a thread's registers hold,
thousands of repeats of one id, minibatches that are empty, tiny or large enough for the larger tiles — against the oracle; and the one-call
hop, whose sampler counts the classes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture
def ctx():
    from graph_sampling_b200 import ops
    c = ops.Context()
    c.set_option("relabel_path", 4)
    yield c


def check(oracle, got, seeds, sp, edges, ep):
    uniq, up, rel = (t.cpu().numpy() for t in got[:3])
    assert up[0] == 0 and up[-1] == len(uniq) and len(rel) == ep[-1]
    for b in range(len(sp) - 1):
        e = edges[ep[b]:ep[b + 1]]
        if sp[b + 1] - sp[b] + len(e) == 0:
            assert up[b] == up[b + 1]
            continue
        want, (w_rel,) = oracle.unique_relabel([seeds[sp[b]:sp[b + 1]], e], [e])
        np.testing.assert_array_equal(uniq[up[b]:up[b + 1]], want)
        np.testing.assert_array_equal(rel[ep[b]:ep[b + 1]], w_rel)


@pytest.mark.parametrize("nodes,sizes,kind", [
    (1, [(1, 40), (0, 3)], "plain"), (16_384, [(100, 20_000), (0, 0), (3, 0)], "plain"), (16_385, [(100, 20_000)] * 3, "edges"),
    (50_000, [(7, 9)] * 900 + [(0, 0)] * 20, "plain"), (300_000, [(1000, 700_000), (10, 100)], "plain"),
    (40_000, [(50, 30_000), (0, 9000)], "one"), (100_000, [(500, 60_000), (20, 4000)], "beyond"),
    (4_161_536, [(30, 5000), (1, 9000)], "edges"), (4_177_920, [(30, 5000)], "plain")])
def test_batched_relabel(oracle, ctx, nodes, sizes, kind):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(nodes + len(sizes))
    sp, ep = (np.concatenate([[0], np.cumsum([s[i] for s in sizes])]) for i in (0, 1))
    seeds, edges = rng.integers(0, nodes, sp[-1]), rng.integers(0, nodes, ep[-1])
    if kind == "edges":
        ends = np.array([v for v in (16_383, 16_384, 32_767, nodes - 1, 0) if v < nodes])
        edges[::2] = rng.choice(ends, len(edges[::2]))
    if kind == "one":
        edges[rng.random(len(edges)) < 0.8] = 777
    if kind == "beyond":
        edges[rng.random(len(edges)) < 0.2] += nodes
        edges[::11] = (1 << 32) - 2 - rng.integers(0, 50, len(edges[::11]))
        edges[5] = -1
        from graph_sampling_b200.cabi import GsbError
        with pytest.raises(GsbError):
            ops.batch_csr_relabel(dev(seeds), dev(sp), dev(edges), dev(ep), num_nodes=nodes, ctx=ctx)
        edges[5] = nodes
    got = ops.batch_csr_relabel(dev(seeds), dev(sp), dev(edges), dev(ep), num_nodes=nodes, ctx=ctx)
    check(oracle, got, seeds, sp, edges, ep)


@pytest.mark.parametrize("nodes,k", [(3000, 5), (40_000, 10), (40_000, 20)])   # a fan-out of 20: no counting sampler
def test_hops(oracle, ctx, nodes, k):
    from conftest import make_graph
    from graph_sampling_b200 import ops
    indptr, indices = make_graph(nodes, 20 * nodes, seed=k)
    rng = np.random.default_rng(k)
    sp = np.concatenate([[0], np.cumsum([300, 0, 1, 700, 40])])
    seeds = rng.integers(0, nodes, sp[-1])
    got = ops.sage_sample_batches(dev(indptr), dev(indices), dev(seeds), dev(sp), [k, 3], seed=6, ctx=ctx)
    ctx.set_option("relabel_path", 1)
    want = ops.sage_sample_batches(dev(indptr), dev(indices), dev(seeds), dev(sp), [k, 3], seed=6, ctx=ctx)
    for a, b in zip(got, want):
        for key in ("sub_indptr", "indices", "relabeled", "select_index", "indices_ptr", "frontier", "frontier_ptr"):
            assert torch.equal(a[key], b[key]), key
    hop = {key: got[0][key].cpu().numpy() for key in ("indices", "relabeled", "indices_ptr", "frontier", "frontier_ptr")}
    check(oracle, (got[0]["frontier"], got[0]["frontier_ptr"], got[0]["relabeled"]), seeds, sp, hop["indices"], hop["indices_ptr"])
