"""The single-launch unique + relabel against the oracle, at the sizes where it can go wrong: one item, the edges of a CTA's
items (512, 1 024, ...), the switches of items per thread, the largest call it serves and the first it leaves to the
general form; minibatches that are empty, tiny, ragged, or more numerous than a CTA keeps in shared memory."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# 151 552 items fill the resident grid at one item per thread; every doubling after that at two, four, eight
SIZES = [1, 31, 32, 33, 511, 512, 513, 1024, 1025, 16_333, 151_551, 151_553, 303_105, 606_211, 1_212_417, 1 << 21,
         (1 << 21) + 1]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def ops():
    from graph_sampling_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("spread", [3, 1 << 31])
def test_graph_relabel_matches_oracle(ops, oracle, n, spread):
    rng = np.random.default_rng(n + spread)
    S = int(rng.integers(0, n + 1))
    ids = rng.integers(0, max(1, int(n * spread) if spread == 3 else spread), n).astype(np.int64)
    first, second = ids[:S], ids[S:]
    frontier, (w_rows,) = oracle.unique_relabel([first, second], [second])
    indptr = rng.integers(0, 1 << 40, 77).astype(np.int64)
    bound = int(ids.max()) + 1 if spread == 3 else 0     # the direct-address table; without a bound the hash table
    assert np.array_equal(ops.graph_unique(dev(first), dev(second), id_bound=max(1, bound - 1)).cpu().numpy(), frontier)
    f, rows, cols, copy, ones = ops.graph_relabel(dev(first), dev(second), indptr=dev(indptr), id_bound=bound, ones=True)
    assert ones.numel() == len(second) and bool((ones == 1.0).all())
    assert cols is None and np.array_equal(f.cpu().numpy(), frontier)
    assert np.array_equal(rows.cpu().numpy(), w_rows) and np.array_equal(copy.cpu().numpy(), indptr)
    f, (rel,) = ops.relabel([dev(first), dev(second)], [dev(second)])
    assert np.array_equal(f.cpu().numpy(), frontier) and np.array_equal(rel.cpu().numpy(), w_rows)
    if S > 0:
        at = rng.integers(0, S, n - S).astype(np.int64)
        _, (w_cols,) = oracle.unique_relabel([first, second], [first[at]])
        f, rows, cols, _ = ops.graph_relabel(dev(first), dev(second), cols=dev(at), id_bound=bound)
        assert np.array_equal(f.cpu().numpy(), frontier)
        assert np.array_equal(rows.cpu().numpy(), w_rows) and np.array_equal(cols.cpu().numpy(), w_cols)


def test_ids_beyond_32_bits_take_the_general_form(ops, oracle):
    first = np.array([5, 1 << 40, 5, (1 << 32) - 1], np.int64)
    second = np.array([1 << 40, 7, 5], np.int64)
    frontier, (want,) = oracle.unique_relabel([first, second], [second])
    f, rows, _, _ = ops.graph_relabel(dev(first), dev(second))
    assert ops.graph_relabel(dev(first), dev(second), ones=True)[4].tolist() == [1.0] * len(second)
    assert np.array_equal(f.cpu().numpy(), frontier) and np.array_equal(rows.cpu().numpy(), want)
    with pytest.raises(Exception):
        ops.graph_relabel(dev(np.array([3, -2], np.int64)), dev(second))
    f, _, _, _ = ops.graph_relabel(dev(np.array([3, 3], np.int64)), dev(second[1:]))   # the context is fine afterwards
    assert f.cpu().tolist() == [3, 7, 5]


def test_a_bound_that_does_not_hold_is_withdrawn(ops, oracle):
    """Ids of a rectangular graph lie beyond its number of columns: the first slice that meets one pays a second launch, the
    others, and later slices of the same graph, do not."""
    import graph_sampling_b200.gs as gs
    rng = np.random.default_rng(3)
    indptr, indices = np.arange(1001) * 20, rng.integers(0, 5000, 20_000)
    graph = gs.Matrix().load_csc(dev(indptr), dev(indices))
    launches = ops.default_context().launch_count
    taken, slices = [], [graph[:, dev(np.arange(i, i + 100))] for i in range(3)]
    for i, sub in enumerate(slices):
        seeds, e = np.arange(i, i + 100), indices[i * 20:(i + 100) * 20]
        want, (want_rows,) = oracle.unique_relabel([seeds, e], [e])
        before = launches()
        frontier, _, _, rows, _, _, fmt = sub._graph._CAPI_relabel()
        taken.append(launches() - before)
        assert fmt == "coo" and np.array_equal(frontier.cpu().numpy(), want) and np.array_equal(rows.cpu().numpy(), want_rows)
        assert np.array_equal(sub._graph._CAPI_all_valid_node().cpu().numpy(), want)
    assert taken == [2, 1, 1]
    square = gs.Matrix().load_csc(dev(indptr), dev(indices % 1000))   # another graph's bound is its own
    square[:, dev(np.arange(100))]._graph._CAPI_relabel()
    assert square._graph._id_bound.value == 1000 and graph._graph._id_bound.value == 0


@pytest.mark.parametrize("G,mean", [(1, 700), (2, 1), (7, 90_000), (40, 3000), (1500, 4), (3000, 300)])
def test_batched_relabel_matches_oracle(ops, oracle, G, mean):
    rng = np.random.default_rng(G * 31 + mean)
    ns, ne = rng.integers(0, mean + 1, G), rng.integers(0, 2 * mean + 1, G)
    ns[rng.random(G) < 0.2] = 0
    ne[rng.random(G) < 0.2] = 0
    ns[0] = max(ns[0], 1)
    sp, ep = np.concatenate([[0], np.cumsum(ns)]), np.concatenate([[0], np.cumsum(ne)])
    seeds, edges = rng.integers(0, 3 * mean + 1, sp[-1]), rng.integers(0, 3 * mean + 1, ep[-1])
    f, fp, rel, _ = ops.batch_csr_relabel(dev(seeds), dev(sp), dev(edges), dev(ep))
    again = ops.batch_csr_relabel(dev(seeds), dev(sp), dev(edges), dev(ep), num_nodes=3 * mean + 1)
    assert all(torch.equal(a, b) for a, b in zip((f, fp, rel), again))
    f, fp, rel = f.cpu().numpy(), fp.cpu().numpy(), rel.cpu().numpy()
    assert fp[0] == 0 and fp[-1] == len(f) and len(rel) == ep[-1]
    for b in range(G):
        e = edges[ep[b]:ep[b + 1]]
        if ns[b] + ne[b] == 0:
            assert fp[b] == fp[b + 1]
            continue
        want, (w_rel,) = oracle.unique_relabel([seeds[sp[b]:sp[b + 1]], e], [e])
        assert np.array_equal(f[fp[b]:fp[b + 1]], want) and np.array_equal(rel[ep[b]:ep[b + 1]], w_rel)


def test_mailbox_tags_wrap(ops):
    """The sizes of a call reach the host in words tagged with one of 65 535 numbers.  A batched call leaves two of them, the
    others one: the second must not be taken from the batched call that had the same number before."""
    ctx, few = ops.Context(), dev(np.arange(32) % 7)
    ptr = dev(np.array([0, 8, 16]))
    calls = [(edges, dev(np.array([0, 400, edges])), dev(np.arange(edges) % 50)) for edges in range(1000, 1005)]
    torch.cuda.synchronize()
    for edges, iptr, ids in calls:
        _, _, rel, _ = ops.batch_csr_relabel(few[:16], ptr, ids, iptr, ctx=ctx)
        assert rel.numel() == edges
        for _ in range(65_534):
            ops.tensor_unique(few, ctx=ctx)


def test_epochs_wrap(ops, oracle):
    """2 047 calls use up the epochs of the table; results stay right across the wrap."""
    rng = np.random.default_rng(1)
    ids = rng.integers(0, 40, 64).astype(np.int64)
    want, _ = oracle.unique_relabel([ids], [])
    d = dev(ids)
    for i in range(2100):
        got, direct = ops.tensor_unique(d), ops.graph_unique(d, d, id_bound=40)
    assert np.array_equal(got.cpu().numpy(), want) and np.array_equal(direct.cpu().numpy(), want)
