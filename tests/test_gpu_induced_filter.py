"""The one-launch induced subgraph at the sizes where it can go wrong: tiles of 4 096 edges that end at and inside columns,
thousands of short and empty columns in a tile, no and all edges kept, repeated row ids, more rows than the shared-memory
filter takes, ids beyond the graph — against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("deg,rows", [
    ([4096, 1, 4095], "some"), ([4095, 4097, 0, 3], "some"), ([1] * 9000, "some"), ([0] * 2000 + [5] + [0] * 3000 + [2], "some"),
    ([30_000] * 11, "none"), ([3, 0, 700, 12] * 500, "all"), ([50] * 40_000, "many"), ([300] * 3000, "repeated")])
def test_induced_subgraph(oracle, deg, rows):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(len(deg) + len(rows))
    n = max(len(deg), 400_000)
    degree = np.zeros(n, np.int64)
    cols = rng.permutation(n)[:len(deg)]
    degree[cols] = deg
    indptr = np.concatenate([[0], np.cumsum(degree)])
    indices = rng.integers(0, n, indptr[-1])
    w = rng.random(indptr[-1], dtype=np.float32)
    count = {"some": n // 20, "none": 1, "all": n, "many": 300_000, "repeated": 5000}[rows]
    ids = rng.permutation(n)[:count]
    if rows == "none":
        ids = np.array([n + 5])
    if rows == "repeated":
        ids = np.concatenate([ids, ids[::2], [n + 7, 1 << 33]])
    want = oracle.col_row_slice(indptr, indices, cols, ids)
    got = [t.cpu().numpy() for t in ops.csc_col_row_slicing(dev(indptr), dev(indices), dev(cols), dev(ids), data=dev(w))]
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    assert np.array_equal(got[3], w[want[2]])
