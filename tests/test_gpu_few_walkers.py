"""Walks at the sizes where the walkers per warp change (148 SMs x 32 warps x 1, 2, 4, 8, 16) and where blocks of four steps end, on
one graph and along a metapath, against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
WARPS = 148 * 32


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("W,L", [(1, 0), (1, 1), (2, 3), (33, 4), (WARPS, 5), (WARPS + 1, 8), (2 * WARPS + 1, 9),
                                 (4 * WARPS + 1, 3), (8 * WARPS + 1, 2), (16 * WARPS, 6), (16 * WARPS + 1, 6)])
def test_walk(oracle, hub_graph, W, L, layout):
    from graph_sampling_b200 import ops
    indptr, indices = hub_graph
    n = len(indptr) - 1
    starts = np.random.default_rng(W + L).integers(0, n, W)
    starts[::7] = -1   # a walker without a start stays where it is
    want = oracle.random_walk(indptr, indices, starts, L, seed=21, layout=layout, walker_offset=3)
    got = ops.fused_random_walk(dev(starts), L, dev(indices), dev(indptr), seed=21, layout=layout, walker_offset=3)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("W", [WARPS, WARPS + 1, 16 * WARPS + 1])
def test_metapath(oracle, hub_graph, W):
    from graph_sampling_b200 import ops
    indptr, indices = hub_graph
    rel = [(indptr, indices), (indptr, indices[::-1].copy())]
    starts = np.random.default_rng(W).integers(0, len(indptr) - 1, W)
    path = [0, 1, 1, 0, 1]
    want = oracle.metapath_random_walk(rel, path, starts, seed=4, layout=0, walker_offset=0)
    got = ops.fused_metapath_random_walk(dev(starts), path, [(dev(a), dev(b)) for a, b in rel], seed=4, layout=0)
    np.testing.assert_array_equal(got.cpu().numpy().reshape(-1), np.asarray(want).reshape(-1))
