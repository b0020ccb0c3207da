"""Uniform sampler whose picks change lanes between the draw and the read: columns, edge data and edge ids of every pick against the
oracle, warps that are full, ragged and empty, and minibatches that end inside a warp while buckets are counted."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def graph(low, high, nodes=3000):
    rng = np.random.default_rng(high)
    degree = rng.integers(low, high, nodes)
    degree[64:96] = 0                       # a warp without a pick when every column is sampled
    indptr = np.concatenate([[0], np.cumsum(degree)])
    return indptr, rng.integers(0, nodes, indptr[-1])


@pytest.mark.parametrize("replace", [False, True])
@pytest.mark.parametrize("k", [1, 4, 5, 7, 8, 10, 13, 16])
@pytest.mark.parametrize("low,high", [(0, 8), (20, 60)])
def test_columns_and_data_of_the_picks(oracle, low, high, k, replace):
    from graph_sampling_b200 import ops
    indptr, indices = graph(low, high)
    rng = np.random.default_rng(k)
    data, e_ids = rng.random(len(indices)).astype(np.float32), rng.permutation(len(indices))
    want = oracle.sample_uniform(indptr, indices, None, k, replace, seed=k, with_coo=True)
    for ids in (None, e_ids):
        got = ops.csc_col_sampling(dev(indptr), dev(indices), k, replace, with_coo=True, seed=k, data=dev(data),
                                   e_ids=None if ids is None else dev(ids))
        for w, g in zip(want, got):
            np.testing.assert_array_equal(g.cpu().numpy(), w)
        np.testing.assert_array_equal(got[4].cpu().numpy(), data[want[3] if ids is None else ids[want[3]]])


@pytest.mark.parametrize("path", [3, 4])
@pytest.mark.parametrize("batch", [5, 32, 45])
def test_bucket_counts_of_minibatches_that_share_a_warp(oracle, path, batch):
    from graph_sampling_b200 import ops
    indptr, indices = graph(0, 40)
    rng = np.random.default_rng(batch)
    G = 50
    seeds = np.concatenate([rng.permutation(3000)[:batch] for _ in range(G)])
    ptr = np.arange(G + 1) * batch
    ctx = ops.Context()
    ctx.set_option("relabel_path", path)
    hop = ops.sage_sample_batches(dev(indptr), dev(indices), dev(seeds), dev(ptr), [10], seed=3, ctx=ctx)[0]
    want = oracle.sample_uniform(indptr, indices, seeds, 10, False, seed=3)
    np.testing.assert_array_equal(hop["indices"].cpu().numpy(), want[2])
    sub, frontier, fptr, rel = want[0], hop["frontier"].cpu().numpy(), hop["frontier_ptr"].cpu().numpy(), hop["relabeled"].cpu().numpy()
    for b in range(G):
        e = want[2][sub[ptr[b]]:sub[ptr[b + 1]]]
        unique, (w_rel,) = oracle.unique_relabel([seeds[ptr[b]:ptr[b + 1]], e], [e])
        np.testing.assert_array_equal(frontier[fptr[b]:fptr[b + 1]], unique)
        np.testing.assert_array_equal(rel[sub[ptr[b]]:sub[ptr[b + 1]]], w_rel)
