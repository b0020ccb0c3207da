"""Calls of one context on several streams in turn: a call comes behind the one before it although that returned with its size
while its last kernel was still running, or without waiting at all."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def ops():
    from graph_sampling_b200 import ops as _ops
    return _ops


def test_scratch_is_not_shared_by_calls_in_flight(ops, oracle):
    rng = np.random.default_rng(1)
    E, keys = 300_000, 200_000
    ids = [rng.integers(0, 400_000, 1_500_000) for _ in range(2)]
    edges = [(rng.integers(0, keys, E), rng.integers(0, 1 << 40, E)) for _ in range(2)]
    unique = [oracle.unique_relabel([x], [])[0] for x in ids]
    order = [np.argsort(key, kind="stable") for key, _ in edges]
    d_ids, d_edges = [dev(x) for x in ids], [(dev(key), dev(other)) for key, other in edges]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    ctx, got = ops.Context(), []
    for turn in range(12):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                key, other = d_edges[i]
                got.append((i, ops.tensor_unique(d_ids[i], ctx=ctx), ops.coo2csc(other, key, keys, False, ctx=ctx)))
                if turn % 2:   # the next stream begins with a conversion that nobody has waited for
                    got.append((1 - i, ops.tensor_unique(d_ids[1 - i], ctx=ctx), None))
    torch.cuda.synchronize()
    ctx.check_device()
    for i, u, conversion in got:
        assert np.array_equal(u.cpu().numpy(), unique[i])
        if conversion is not None:
            key, other = edges[i]
            indptr, rows, perm = (t.cpu().numpy() for t in conversion)
            assert np.array_equal(perm, order[i]) and np.array_equal(rows, other[order[i]])
            assert np.array_equal(indptr, np.concatenate([[0], np.cumsum(np.bincount(key, minlength=keys))]))
