"""Which uniform samples are taken by windows of the edges: three launches, one for one pass, on both sides of every line of the rule.
The results are the same either way."""
import functools

import pytest
import torch

pytestmark = pytest.mark.gpu


@functools.lru_cache(1)
def graph(edges):
    gen = torch.Generator("cuda").manual_seed(7)
    columns = edges // 20
    indptr = torch.arange(columns + 1, device="cuda") * 20
    return indptr, torch.randint(0, columns, (edges,), generator=gen, device="cuda")


@pytest.mark.parametrize("edges,k,columns,windows", [
    (31_000_000, 5, 6_199_000, False), (31_000_000, 5, 6_200_000, True),       # up to four windows: a pick per edge,
    (31_000_000, 10, 3_449_000, False), (31_000_000, 10, 3_450_000, True),     # with more picks by the edges,
    (19_000_000, 10, 16_000_000, False),
    (31_000_000, 8, 15_500_000, False), (31_000_000, 12, 12_000_000, False),   # and never with so many
    (34_000_000, 5, 2_399_000, False), (34_000_000, 5, 2_400_000, True),       # five windows
    (34_000_000, 10, 1_999_000, False), (34_000_000, 10, 2_000_000, True),
    (34_000_000, 8, 4_999_000, False), (34_000_000, 8, 5_000_000, True),
    (34_000_000, 16, 8_500_000, False)])
def test_lines_of_the_rule(edges, k, columns, windows):
    from graph_sampling_b200 import ops
    indptr, indices = graph(edges)
    seeds = torch.randint(0, edges // 20, (columns,), generator=torch.Generator("cuda").manual_seed(k), device="cuda")
    auto, plain = ops.Context(), ops.Context()
    plain.set_option("sample_path", 1)
    got = ops.fused_csc_col_slicing_sampling(indptr, indices, seeds, k, False, seed=2, ctx=auto)
    assert auto.launch_count() == (3 if windows else 1)
    want = ops.fused_csc_col_slicing_sampling(indptr, indices, seeds, k, False, seed=2, ctx=plain)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
