"""The slice copy at the sizes where it can go wrong: stretches that end inside, at and between columns,
columns much longer and much shorter than a stretch, more (empty) columns in it than its window holds, every optional
output, and the batched form with encoded ids — against numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


SHAPES = {"one": [1], "exact": [1024, 1024], "off_by_one": [1023, 1, 1, 1025], "hub": [0, 50_001, 3], "short": [3] * 5000,
          "empty_runs": [2] + [0] * 3000 + [5] + [0] * 700 + [1, 1, 1], "mixed": [7, 0, 900, 0, 0, 2100, 1, 40] * 60,
          "all_empty": [0] * 70, "stretches": [7, 0, 900, 0, 0, 2100, 1, 40] * 700, "many": [3, 0, 0, 4] * 200_000}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("indirect", [False, True])
def test_column_slice(shape, indirect):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(len(shape))
    deg = np.array(SHAPES[shape], np.int64)
    indptr = np.concatenate([[0], np.cumsum(deg)])
    E = int(indptr[-1])
    indices, data = rng.integers(0, 1 << 33, E), rng.random(E, dtype=np.float32)
    e_ids = rng.permutation(E).astype(np.int64) if indirect else None
    seeds = rng.permutation(len(deg)) if indirect else np.arange(len(deg))
    want = np.concatenate([np.arange(indptr[c], indptr[c + 1]) for c in seeds]).astype(np.int64)
    got = ops.csc_col_slicing(dev(indptr), dev(indices), dev(seeds) if indirect else None, True, data=dev(data),
                              e_ids=None if e_ids is None else dev(e_ids))
    sub_indptr, col, idx, select, out = [t.cpu().numpy() for t in got]
    assert np.array_equal(sub_indptr, np.concatenate([[0], np.cumsum(deg[seeds])]))
    assert np.array_equal(select, want) and np.array_equal(idx, indices[want])
    assert np.array_equal(col, np.repeat(np.arange(len(deg)), deg[seeds]))
    assert np.array_equal(out, data[e_ids[want]] if indirect else data[want])
    lean = ops.col_slice(dev(indptr), dev(indices), dev(seeds), False)
    assert lean[1] is None and lean[3] is None and np.array_equal(lean[2].cpu().numpy(), indices[want])
    ptr = np.array([0, len(seeds) // 3, len(seeds) // 3, len(seeds)])
    batch = np.repeat(np.arange(3), np.diff(ptr))
    got = ops.batch_csc_col_slicing(dev(indptr), dev(indices), dev(seeds), dev(ptr), 1000, True, True)
    assert np.array_equal(got[2].cpu().numpy(), indices[want] + 1000 * np.repeat(batch, deg[seeds]))
