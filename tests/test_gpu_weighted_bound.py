"""Weighted sampling where the k best of a column are found behind a bound, against the oracle: columns on both sides of 32, 64 and 128
edges and longer, fan-outs on both sides of half the lanes, and weights that leave few or all entries at the bound."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def weights(rng, kind, n):
    if kind == "random":
        return rng.random(n)
    if kind == "few":
        return np.where(rng.random(n) < 0.1, rng.random(n), 0.0)
    if kind == "odd":
        return rng.choice([0.0, -1.0, np.nan, np.inf, 1e-38, 1e-45, 3e38, 1.0], n)
    return np.full(n, float(kind))


@pytest.mark.parametrize("kind", ["random", "few", "odd", "0", "inf"])
@pytest.mark.parametrize("k", [1, 4, 5, 8, 9, 16, 17, 32])
def test_against_the_oracle(oracle, k, kind):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(k)
    degree = np.concatenate([[0, 1, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 512, 513, 1024, 1100, 3000], rng.integers(1, 140, 900)])
    indptr = np.concatenate([[0], np.cumsum(degree)])
    indices = rng.integers(0, 5000, indptr[-1])
    probs = weights(rng, kind, len(indices)).astype(np.float32)
    want = oracle.sample_weighted(indptr, indices, probs, None, k, False, seed=k, with_coo=True)
    got = ops.csc_col_sampling_probs(dev(indptr), dev(indices), dev(probs), k, False, seed=k)
    for w, g in zip(want, got):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
