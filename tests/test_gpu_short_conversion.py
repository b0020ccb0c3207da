"""The conversion of a short edge list at its edges: one edge, a warp's and a CTA's share of the keys, one key per CTA, the most keys
and edges it takes and the first beyond, all edges on the first, the last or one key in the middle, the edges
of a CTA and the keys at which it sorts by one and by two digits, keys out of range."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("E,keys,kind", [
    (1, 1, "uniform"), (2, 148, "uniform"), (31, 149, "uniform"), (1024, 147, "uniform"), (1025, 296, "skewed"),
    (26_624, 5, "uniform"), (26_624, 1, "uniform"), (26_623, 4737, "skewed"), (26_624, 8192 * 148, "uniform"),
    (26_624, 8192 * 148, "skewed"), (26_624, 8192 * 148 + 1, "uniform"), (26_625, 1000, "uniform"), (26_000, 100_003, "first"),
    (26_000, 100_003, "last"), (26_624, 100_003, "middle"), (777, 1_000_000, "uniform"),
    (1023, 1, "uniform"), (1024, 1, "uniform"), (2000, 1, "uniform"), (26_000, 148 * 128, "skewed"), (26_000, 148 * 129, "skewed")])
def test_stable_sort(E, keys, kind):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(E + keys)
    key = {"uniform": lambda: rng.integers(0, keys, E), "first": lambda: np.zeros(E, np.int64), "last": lambda: np.full(E, keys - 1),
           "middle": lambda: np.full(E, keys // 2),
           "skewed": lambda: np.minimum((keys * rng.random(E) ** 6).astype(np.int64), keys - 1)}[kind]()
    other = rng.integers(0, 1 << 40, E)
    indptr, out, perm = (t.cpu().numpy() for t in ops.coo2csc(dev(other), dev(key), keys, False))
    want = np.argsort(key, kind="stable")
    np.testing.assert_array_equal(perm, want)
    np.testing.assert_array_equal(out, other[want])
    np.testing.assert_array_equal(indptr, np.concatenate([[0], np.cumsum(np.bincount(key, minlength=keys))]))


def test_keys_out_of_range_count_as_key_0():
    from graph_sampling_b200 import ops
    from graph_sampling_b200.cabi import GsbError
    ctx = ops.Context()
    key = np.arange(5000) % 700
    key[[3, 4999]] = -1, 700
    indptr, out, perm = (t.cpu().numpy() for t in ops.coo2csc(dev(np.arange(5000)), dev(key), 700, False, ctx=ctx))
    with pytest.raises(GsbError) as e:
        ctx.check_device()
    assert e.value.status == -8
    key[[3, 4999]] = 0
    np.testing.assert_array_equal(perm, np.argsort(key, kind="stable"))
    np.testing.assert_array_equal(indptr, np.concatenate([[0], np.cumsum(np.bincount(key, minlength=700))]))
