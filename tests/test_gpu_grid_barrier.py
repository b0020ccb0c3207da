"""Cooperative kernels whose grid barrier runs out of polls (GSB_OPT_MAX_POLLS = 1, so that the first CTAs to arrive give up):
the call reports it, what it leaves behind lies within its buffers and is a result that later kernels can read, and the
context works as before once the error is read.  A call that gets through all the same has to be right."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TIMEOUT = -5
PAD = 64


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def ops():
    from graph_sampling_b200 import ops as _ops
    return _ops


def as_numpy(x):
    if isinstance(x, (tuple, list)):
        return [as_numpy(y) for y in x]
    return x.cpu().numpy() if isinstance(x, torch.Tensor) else x


def same(a, b):
    if isinstance(a, list):
        return len(a) == len(b) and all(same(x, y) for x, y in zip(a, b))
    return np.array_equal(a, b) if a is not None else b is None


def run_out(ops, call, left_behind=None):
    """Calls until the barrier has run out a few times, then again with the usual limit."""
    from graph_sampling_b200.cabi import GsbError
    ctx = ops.Context()
    want = as_numpy(call(ctx))
    ctx.check_device()
    usual, expired = ctx.get_option("max_polls"), 0
    ctx.set_option("max_polls", 1)
    for _ in range(200):
        got = None
        try:
            got = as_numpy(call(ctx))
            ctx.check_device()
        except GsbError as e:
            assert e.status == TIMEOUT
            expired += 1
            if got is not None and left_behind is not None:
                left_behind(got)
            if expired == 5:
                break
        else:
            assert same(got, want)
    assert expired > 0
    ctx.set_option("max_polls", usual)
    for _ in range(2):
        assert same(as_numpy(call(ctx)), want)
        ctx.check_device()


def graph(n, m, seed):
    from tests.conftest import make_graph
    return tuple(dev(a) for a in make_graph(n, m, seed=seed))


@pytest.mark.parametrize("E,keys", [(300_001, 2000), (300_001, 1_000_000), (1_000_003, 5_000_000)])   # one, two, three digits
def test_conversion(ops, E, keys):
    rng = np.random.default_rng(E + keys)
    key, other = dev(rng.integers(0, keys, E)), dev(rng.integers(0, 1 << 40, E))

    def call(ctx):
        sizes = (keys + 1, E, E)
        out = [torch.full((n + PAD,), -7, dtype=torch.int64, device="cuda") for n in sizes]
        ctx.check(ctx.lib.gsb_coo2csc(ctx.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), key.data_ptr(),
                                      other.data_ptr(), E, keys, 0, *(t.data_ptr() for t in out)), "gsb_coo2csc")
        assert all(bool((t[n:] == -7).all()) for t, n in zip(out, sizes))
        return [t[:n] for t, n in zip(out, sizes)]

    everything = other.cpu().numpy()

    def left_behind(got):
        indptr, rows, perm = got
        assert indptr[0] == 0 and np.all(indptr[1:] == E)
        assert perm.min() >= 0 and perm.max() < E and np.isin(rows, everything).all()

    run_out(ops, call, left_behind)


@pytest.mark.parametrize("k", [7, 4096])
def test_list_sampling(ops, k):
    N = 1_000_000
    rng = np.random.default_rng(k)
    data, probs = dev(rng.permutation(N)), dev(rng.random(N, dtype=np.float32))

    def left_behind(got):
        assert np.array_equal(got[1], np.arange(k)) and np.array_equal(got[0], data[:k].cpu().numpy())

    run_out(ops, lambda ctx: ops.list_sampling(data, k, False, probs, seed=3, ctx=ctx), left_behind)


@pytest.mark.parametrize("n", [200_000, 2_000_000])
@pytest.mark.parametrize("bound", [0, 500_000])
def test_unique_and_relabel(ops, n, bound):
    ids = dev(np.random.default_rng(n).integers(0, 500_000, n))
    first, second = ids[:n // 3].contiguous(), ids[n // 3:].contiguous()
    run_out(ops, lambda ctx: ops.graph_relabel(first, second, ctx=ctx, id_bound=bound))


@pytest.mark.parametrize("num_nodes", [0, 50_000])
def test_batched_relabel(ops, num_nodes):
    rng = np.random.default_rng(7)
    sp, ep = np.arange(41) * 500, np.arange(41) * 12_000
    seeds, edges = dev(rng.integers(0, 50_000, sp[-1])), dev(rng.integers(0, 50_000, ep[-1]))
    d_sp, d_ep = dev(sp), dev(ep)
    run_out(ops, lambda ctx: ops.batch_csr_relabel(seeds, d_sp, edges, d_ep, ctx=ctx, num_nodes=num_nodes)[:3])

    def queued(ctx):   # no wait for the sizes: the totals are those of the device
        _, ptr, rel, _ = ops.batch_csr_relabel(seeds, d_sp, edges, d_ep, ctx=ctx, num_nodes=num_nodes, sync=False,
                                               indices_count=int(ep[-1]))
        return ptr, rel

    run_out(ops, queued, lambda got: np.testing.assert_array_equal(got[0], 0) or np.testing.assert_array_equal(got[1], -1))


@pytest.mark.parametrize("k", [5, 16, 40])
@pytest.mark.parametrize("replace", [False, True])
def test_weighted_sampling(ops, hub_graph, k, replace):
    indptr, indices = (dev(a) for a in hub_graph)
    probs = torch.rand(indices.numel(), generator=torch.Generator("cuda").manual_seed(4), device="cuda") + 0.01
    # read in place from host memory: the CTAs' columns arrive one after the other
    columns = torch.from_numpy(np.random.default_rng(k).integers(0, len(hub_graph[0]) - 1, 400_000)).pin_memory()
    run_out(ops, lambda ctx: ops.csc_col_sampling_probs(indptr, indices, probs, k, replace, seed=8, column_ids=columns, ctx=ctx))


def test_induced_subgraph(ops):
    indptr, indices = graph(100_000, 2_000_000, 6)
    nodes = dev(np.random.default_rng(2).permutation(100_000)[:20_000])
    offsets, _, sliced, _ = ops.csc_col_slicing(indptr, indices, nodes, False)
    S, D = nodes.numel(), sliced.numel()

    def call(ctx, wait=True):   # the second step of ops.csc_col_row_slicing; the first counts with a look-back of its own
        out = [torch.full((n + PAD,), -7, dtype=torch.int64, device="cuda") for n in (S + 1, D, D)]
        nnz = ctypes.c_int64(0)
        ctx.check(ctx.lib.gsb_col_row_slice(ctx.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                            indptr.data_ptr(), indices.data_ptr(), indptr.numel() - 1, nodes.data_ptr(), S,
                                            offsets.data_ptr(), D, nodes.data_ptr(), S, None, None, 1, 0, 1,
                                            *(t.data_ptr() for t in out), None, None, None,
                                            ctypes.byref(nnz) if wait else None), "gsb_col_row_slice")
        assert all(bool((t[n:] == -7).all()) for t, n in zip(out, (S + 1, D, D)))
        return [t[:n] for t, n in zip(out, (S + 1, D, D))]

    run_out(ops, call)
    run_out(ops, lambda ctx: call(ctx, wait=False), lambda got: np.testing.assert_array_equal(got[0], 0))
