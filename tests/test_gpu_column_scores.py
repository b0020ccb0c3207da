"""Scores and weighted draws column by column: the register sort of short columns and its size classes, the slices of long
ones, the running sums of draws with replacement, and the dot product that holds a column's row, at the edges of their
classes against the CPU oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 5, 16, 17, 31, 32, 33, 40, 41, 63, 64, 65, 100, 127, 128, 129, 255, 256, 257, 513, 2047, 2048, 2049, 4097, 9001]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def ops():
    from graph_sampling_b200 import ops as m
    return m


@pytest.fixture(scope="module")
def columns():
    rng = np.random.default_rng(7)
    n = 10_000
    indptr = np.concatenate([[0], np.cumsum(DEGREES)]).astype(np.int64)
    indices = rng.integers(0, n, indptr[-1]).astype(np.int64)
    probs = rng.random(indptr[-1]).astype(np.float32)
    probs[rng.random(len(probs)) < 0.1] = 0.0             # tied keys: the smaller position ranks first
    for c, value in ((12, 0.0), (15, np.inf), (19, 0.0), (24, 0.0)):
        probs[indptr[c]:indptr[c + 1]] = value
    return indptr, indices, probs


# column counts on both sides of where a CTA takes 1, 2, 4, 8 and 32 columns
@pytest.mark.parametrize("S", [1, 27, 2368, 2369, 4737, 9473, 18944, 20011])
@pytest.mark.parametrize("k,replace", [(1, False), (16, False), (32, False), (40, False), (100, False), (9, True), (40, True)])
def test_weighted_columns_of_every_class(ops, oracle, columns, S, k, replace):
    indptr, indices, probs = columns
    rng = np.random.default_rng(S + k)
    seeds = rng.integers(0, 19, S).astype(np.int64)       # short ones, and a few of each long class
    some = rng.integers(0, S, 30)
    seeds[some] = rng.integers(19, len(DEGREES), len(some))
    want = oracle.sample_weighted(indptr, indices, probs, seeds, k, replace, seed=3, with_coo=True)
    got = ops.csc_col_sampling_probs(dev(indptr), dev(indices), dev(probs), k, replace, with_coo=True, seed=3,
                                     column_ids=dev(seeds))
    for w, g in zip(want, got[:4]):
        assert np.array_equal(w, g.cpu().numpy())


@pytest.mark.parametrize("E", [1, 15, 16, 17, 333])
@pytest.mark.parametrize("F", [4, 32, 36, 64, 68, 128, 132, 256, 260, 512, 516])
def test_dot_with_a_held_row(ops, oracle, E, F):
    rng = np.random.default_rng(E + F)
    col = np.sort(rng.integers(0, 40, E)).astype(np.int64)
    row = rng.integers(0, 200, E).astype(np.int64)
    e_ids = rng.permutation(E).astype(np.int64)
    src, dst = rng.standard_normal((200, F)).astype(np.float32), rng.standard_normal((40, F)).astype(np.float32)
    scale = np.abs(src[row] * dst[col]).sum(1, keepdims=True)
    for lhs, rhs, lt, rt, ids in ((src, dst, 0, 2, None), (dst, src, 2, 0, e_ids)):
        want = oracle.sddmm_coo("dot", row, col, lhs, rhs, lt, rt, e_ids=ids)
        out = torch.zeros(E, 1, device="cuda")
        ops.sddmm("dot", dev(lhs), dev(rhs), out, lt, rt, dev(row), dev(col), e_ids=None if ids is None else dev(ids))
        at = np.arange(E) if ids is None else ids
        assert np.all(np.abs(out.cpu().numpy()[at] - want[at]) <= 1e-5 * scale + 1e-7)
