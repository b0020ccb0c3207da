"""List sampling without replacement where its forms change: keys in registers up to 8 192 items per CTA, winners ranked by all CTAs up
to 192 per CTA and sorted by one beyond, with ties, without weights, with few and no positive weights — against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("weights", [None, "random", "few", "none", "equal", "nan"])
@pytest.mark.parametrize("N,k", [(193, 192), (4096, 193), (4097, 384), (4097, 385), (90_112, 4096), (86_016, 4096), (2 * 4096, 384),
                                 (1_212_416, 100), (1_212_417, 4096)])
def test_against_oracle(oracle, N, k, weights):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(N + k)
    data = rng.permutation(N)
    probs = None
    if weights is not None:
        probs = rng.random(N, dtype=np.float32)
        if weights == "few":
            probs[rng.random(N) < 0.97] = 0
        if weights == "none":
            probs[:] = 0
        if weights == "equal":
            probs[:] = 1
        if weights == "nan":
            probs[::3], probs[1::3] = np.nan, -1
    want = oracle.list_sample(data, probs, k, False, seed=5)
    got = ops.list_sampling(dev(data), k, False, None if probs is None else dev(probs), seed=5)
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b.cpu().numpy())
