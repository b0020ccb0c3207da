"""Uniform sampling by windows of the edges against the oracle: edges of tiles and of windows, hubs and empty columns, ids that 32
bits don't hold, bad seeds, buffers that are too small, and the hop that counts buckets along the way."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(5)
    degree = rng.integers(0, 60, 4000)
    degree[::7], degree[11], degree[3999] = 0, 30_000, 5000      # a hub over several windows, the last column
    indptr = np.concatenate([[0], np.cumsum(degree)])
    return indptr, rng.integers(0, 4000, indptr[-1])


def windows():
    from graph_sampling_b200 import ops
    ctx = ops.Context()
    ctx.set_option("sample_path", 2)
    return ctx


@pytest.mark.parametrize("replace", [False, True])
@pytest.mark.parametrize("k", [1, 3, 5, 6, 10, 11, 16])
def test_against_the_oracle(oracle, graph, k, replace):
    from graph_sampling_b200 import ops
    indptr, indices = graph
    rng = np.random.default_rng(k)
    for S in (0, 1, 511, 512, 513, 40_000):
        seeds = rng.integers(0, 4000, S)
        want = oracle.sample_uniform(indptr, indices, seeds, k, replace, seed=k)
        got = ops.fused_csc_col_slicing_sampling(dev(indptr), dev(indices), dev(seeds), k, replace, seed=k, ctx=windows())
        for w, g in zip((want[0], want[2], want[3]), got):
            np.testing.assert_array_equal(g.cpu().numpy(), w)


def test_ids_beyond_32_bits_and_no_seeds(oracle, graph):
    from graph_sampling_b200 import ops
    indptr, indices = graph
    indices = indices.copy()
    indices[::5], indices[1::5], indices[2::5] = -1, 2**32 - 1, 2**40 + 3
    want = oracle.sample_uniform(indptr, indices, None, 7, False, seed=3)
    got = ops.csc_col_sampling(dev(indptr), dev(indices), 7, False, with_coo=False, seed=3, ctx=windows())
    np.testing.assert_array_equal(got[0].cpu().numpy(), want[0])
    np.testing.assert_array_equal(got[2].cpu().numpy(), want[2])


def test_bad_seeds_are_empty_columns(oracle, graph):
    from graph_sampling_b200 import ops
    from graph_sampling_b200.cabi import GsbError
    indptr, indices = graph
    seeds, ctx = np.arange(2000) % 1000, windows()
    for bad in (-1, 4000, 2**40):
        seeds[1500] = bad
        with pytest.raises(GsbError) as e:
            ops.fused_csc_col_slicing_sampling(dev(indptr), dev(indices), dev(seeds), 5, False, ctx=ctx)
        assert e.value.status == -8
    seeds[1500] = 0     # column 0 is empty
    want = oracle.sample_uniform(indptr, indices, seeds, 5, False, seed=9)
    got = ops.fused_csc_col_slicing_sampling(dev(indptr), dev(indices), dev(seeds), 5, False, seed=9, ctx=ctx)
    np.testing.assert_array_equal(got[1].cpu().numpy(), want[2])


# hashed buckets, classes of ids (more than 256 counted in shared memory), minibatches that end inside a tile
@pytest.mark.parametrize("path", [3, 4])
@pytest.mark.parametrize("G,batch", [(1, 5000), (37, 123), (400, 3)])
def test_hops_with_bucket_counts(graph, path, G, batch):
    from graph_sampling_b200 import ops
    indptr, indices = graph
    rng = np.random.default_rng(G)
    seeds = np.concatenate([rng.permutation(4000)[:min(batch, 4000)] for _ in range(G)])
    ptr = np.arange(G + 1) * (len(seeds) // G)
    ids = rng.integers(0, 2**31, G)
    out = []
    for sample_path in (1, 2):
        ctx = ops.Context()
        ctx.set_option("sample_path", sample_path)
        ctx.set_option("relabel_path", path)
        for batch_ids in (None, dev(ids)):
            out.append(ops.sage_sample_batches(dev(indptr), dev(indices), dev(seeds), dev(ptr), [5, 10], seed=1, ctx=ctx,
                                               batch_ids=batch_ids))
    for one, two in ((out[0], out[2]), (out[1], out[3])):
        for a, b in zip(one, two):
            for key in a:
                assert torch.equal(a[key], b[key]), key


def test_too_small_a_buffer_is_reported(graph):
    from graph_sampling_b200 import ops
    from graph_sampling_b200.cabi import GsbError
    indptr, indices = graph
    seeds, ctx = np.arange(4000), windows()
    ctx.set_option("relabel_path", 3)
    args = (dev(indptr), dev(indices), dev(seeds), dev(np.array([0, 2000, 4000])), [5])
    ops.sage_sample_batches(*args, seed=1, ctx=ctx, sync=False, size_hints=[(4000, 9000)])
    with pytest.raises(GsbError) as e:
        ctx.check_device()
    assert e.value.status == -4
    whole = ops.sage_sample_batches(*args, seed=1, ctx=ctx)[0]
    other = ops.sage_sample_batches(*args, seed=1)[0]
    assert torch.equal(whole["relabeled"], other["relabeled"]) and torch.equal(whole["frontier"], other["frontier"])


def test_automatic_choice(oracle):
    """20 M edges, 67.5 M picks: just below the rule and just above, the same results."""
    from graph_sampling_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    indptr = torch.arange(1_000_001, device="cuda") * 20
    indices = torch.randint(0, 1_000_000, (20_000_000,), generator=gen, device="cuda")
    for S in (6_749_900, 6_750_100):
        seeds = torch.randint(0, 1_000_000, (S,), generator=gen, device="cuda")
        plain, auto = ops.Context(), ops.Context()
        plain.set_option("sample_path", 1)
        launches = auto.launch_count()
        got = ops.fused_csc_col_slicing_sampling(indptr, indices, seeds, 10, False, seed=2, ctx=auto)
        assert auto.launch_count() - launches == (1 if S < 6_750_000 else 3)
        want = ops.fused_csc_col_slicing_sampling(indptr, indices, seeds, 10, False, seed=2, ctx=plain)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
