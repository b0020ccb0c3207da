"""Forms that want more scratch than the others: what they take of the device's memory, and the call that goes another way where
there is too little left of it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20


class Filled:
    """All but `leave` bytes of the device's free memory are taken."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.block = torch.empty(torch.cuda.mem_get_info()[0] - self.leave, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        del self.block
        torch.cuda.empty_cache()


def test_windows_leave_the_memory_to_the_caller():
    from graph_sampling_b200 import ops
    n, S, k = 100_000, 4_500_000, 10          # 189 MB of scratch; 756 MB of results
    gen = torch.Generator("cuda").manual_seed(4)
    indptr, indices = torch.arange(n + 1, device="cuda") * 20, torch.randint(0, n, (n * 20,), generator=gen, device="cuda")
    seeds = torch.randint(0, n, (S,), generator=gen, device="cuda")

    def call(ctx):
        before = ctx.launch_count()
        got = ops.fused_csc_col_slicing_sampling(indptr, indices, seeds, k, False, seed=3, ctx=ctx)
        return got, ctx.launch_count() - before

    plain, ctx = ops.Context(), ops.Context()
    plain.set_option("sample_path", 1)
    want = [t.cpu() for t in call(plain)[0]]
    ctx.set_option("sample_path", 1)
    call(ctx)                                 # look-back words are there from now on
    ctx.set_option("sample_path", 2)
    with Filled(1300 * MB):                   # less than eight times the scratch is left beside the results
        free = torch.cuda.mem_get_info()[0]
        got, launches = call(ctx)
        assert launches == 1 and all(torch.equal(a.cpu(), b) for a, b in zip(got, want))
        del got
        torch.cuda.empty_cache()
        assert free - torch.cuda.mem_get_info()[0] <= 4 * MB
    free = torch.cuda.mem_get_info()[0]
    for _ in range(64):                       # a size that was refused is not asked for by every call
        got, launches = call(ctx)
    assert launches == 3 and all(torch.equal(a.cpu(), b) for a, b in zip(got, want))
    del got
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert free - torch.cuda.mem_get_info()[0] <= S * (4 * k + 3) + 4 * MB


def test_class_tiles_step_back():
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(5)
    G, nodes = 2000, 200_000                  # 16.4 M items in half-filled tiles: 1.3 GB of scratch, 0.54 in buckets
    sp, ep = np.arange(G + 1) * 1000, np.arange(G + 1) * 7200
    dev = [torch.from_numpy(a).cuda() for a in (rng.integers(0, nodes, sp[-1]), sp, rng.integers(0, nodes, ep[-1]), ep)]

    def call(ctx, path):
        ctx.set_option("relabel_path", path)
        before = ctx.launch_count()
        got = ops.batch_csr_relabel(*dev, num_nodes=nodes, ctx=ctx)[:3]
        return got, ctx.launch_count() - before

    want, in_buckets = call(ops.Context(), 4)
    want = [t.cpu() for t in want]
    ctx = ops.Context()
    with Filled(1250 * MB):
        got, launches = call(ctx, 5)
        assert launches == in_buckets and all(torch.equal(a.cpu(), b) for a, b in zip(got, want))
        del got
    got, launches = [call(ctx, 5) for _ in range(64)][-1]
    assert launches < in_buckets and all(torch.equal(a.cpu(), b) for a, b in zip(got, want))
