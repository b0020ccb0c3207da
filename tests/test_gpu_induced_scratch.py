"""Scratch of the one-launch induced subgraph: at most 12 bytes and a quarter per edge of its columns (and the quarter more that a
growing workspace takes), with the result against torch; positions beyond 32 bits against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("positions", [True, False])
def test_scratch_per_edge(positions):
    from graph_sampling_b200 import ops
    n, deg = 40_000, 900
    gen = torch.Generator("cuda").manual_seed(4)
    indptr = torch.arange(n + 1, device="cuda") * deg
    indices = torch.randint(0, n, (n * deg,), generator=gen, device="cuda")
    cols = torch.arange(n, device="cuda")
    rows = torch.randperm(n, generator=gen, device="cuda")[:1000]
    call = ops.csc_col_row_slicing if positions else ops.col_row_slice
    call(indptr, indices, cols, rows)  # torch's own memory is there from now on
    ctx = ops.Context()
    call(indptr[:2], indices, cols[:1], rows, ctx=ctx)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    out = call(indptr, indices, cols, rows, ctx=ctx)
    torch.cuda.synchronize()
    grown = before - torch.cuda.mem_get_info()[0]
    bound = 1.25 * (12.25 * n * deg + (8 << 20)) + (4 << 20)  # tables and look-back words, the driver's granularity
    assert grown <= bound, (grown, bound)
    place = torch.full((n,), -1, device="cuda").scatter_(0, rows, torch.arange(1000, device="cuda"))
    kept = place[indices] >= 0
    assert torch.equal(out[1], place[indices[kept]])
    assert torch.equal(out[0][1:], torch.cumsum(kept.view(n, deg).sum(1), 0))
    if positions:
        assert torch.equal(out[2], kept.nonzero().squeeze(1))


def test_positions_beyond_32_bits(oracle):
    """Columns that lie behind the first 2^32 edges of the operand, whose positions need their high part."""
    from graph_sampling_b200 import ops
    base, n, deg = (1 << 32) + 5, 3000, 70
    if torch.cuda.mem_get_info()[0] < 8 * (base + n * deg) + (4 << 30):
        pytest.skip("needs 39 GB of device memory")
    rng = np.random.default_rng(8)
    tail = rng.integers(0, n, n * deg)
    cols, rows = rng.permutation(n)[:900], rng.permutation(n)[:1200]
    indices = torch.empty(base + n * deg, dtype=torch.int64, device="cuda")
    indices[base:] = torch.from_numpy(tail).cuda()
    indptr = base + np.arange(n + 1) * deg
    got = ops.csc_col_row_slicing(torch.from_numpy(indptr).cuda(), indices, torch.from_numpy(cols).cuda(), torch.from_numpy(rows).cuda())
    want = oracle.col_row_slice(indptr - base, tail, cols, rows)
    for a, b, shift in zip(want[:3], got, (0, 0, base)):
        np.testing.assert_array_equal(a + shift, b.cpu().numpy())
    del indices, got
    torch.cuda.empty_cache()
