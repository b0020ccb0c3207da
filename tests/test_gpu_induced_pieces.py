"""The one-launch induced subgraph where its columns are taken in pieces: columns around 32 and 64 long, the degree at which the
form changes, empty columns between them, columns longer than a warp's stretch, ids and row ids beyond 32 bits
whose low halves meet, edge data with and without edge ids — against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("permuted", [False, True])
@pytest.mark.parametrize("deg", [[20] * 700, [19] * 700, [31, 32, 33, 64, 65, 1, 0] * 40, [0] * 40 + [2000] + [0] * 40 + [1] * 7,
                                 [150_000, 3, 0, 150_000], [33] * 33, [1000] * 1200])
def test_pieces(oracle, deg, permuted):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(sum(deg) + len(deg))
    n = max(5000, len(deg))
    degree = np.zeros(n, np.int64)
    cols = rng.permutation(n)[:len(deg)]
    degree[cols] = deg
    indptr = np.concatenate([[0], np.cumsum(degree)])
    E = int(indptr[-1])
    indices = rng.integers(0, n, E)
    indices[rng.random(E) < 0.1] += 1 << 32      # the same low half as an id of the graph
    indices[rng.random(E) < 0.1] += 5 << 40
    rows = np.concatenate([rng.permutation(n)[:n // 3], (1 << 32) + rng.permutation(n)[:n // 3]])
    w, e_ids = rng.random(E, dtype=np.float32), rng.permutation(E) if permuted else None
    want = oracle.col_row_slice(indptr, indices, cols, rows)
    got = [t.cpu().numpy() for t in ops.csc_col_row_slicing(dev(indptr), dev(indices), dev(cols), dev(rows), data=dev(w),
                                                            e_ids=None if e_ids is None else dev(e_ids))]
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(got[3], w[want[2]] if e_ids is None else w[e_ids[want[2]]])
