"""Grid barriers of the cooperative kernels and look-back chains of the scans that run out of polls (GSB_OPT_MAX_POLLS = 1, so
that the first CTAs to wait give up): the call reports it, what it leaves behind lies within its buffers and is a result that
later kernels can read, and the context works as before once the error is read.  A call that gets through all the same has to
be right: a wait that was given up anywhere in the call must not go unnoticed."""
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


def pinned(a):
    """Read in place from host memory: what the CTAs wait for arrives one CTA after the other."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def run_out(ops, call, left_behind=None, tries=200, certain=True):
    """Calls until a wait has run out a few times, then again with the usual limit.  certain=False: the CTAs arrive so close to
    each other that no wait may run out, whatever the limit."""
    from graph_sampling_b200.cabi import GsbError
    ctx = ops.Context()
    want = as_numpy(call(ctx))
    ctx.check_device()
    usual, expired = ctx.get_option("max_polls"), 0
    ctx.set_option("max_polls", 1)
    for _ in range(tries):
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
    assert expired > 0 or not certain
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
    # with a table addressed by the id the 200 CTAs of the small call are done with a few reductions each, and a wait is given up
    # only between two arrivals
    run_out(ops, lambda ctx: ops.graph_relabel(first, second, ctx=ctx, id_bound=bound), certain=n > 200_000 or bound == 0)


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
    columns = pinned(np.random.default_rng(k).integers(0, len(hub_graph[0]) - 1, 400_000))
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


# ---- look-back chains ------------------------------------------------------------------------------------------------------
def test_slice_offsets(ops):
    indptr, _ = graph(100_000, 2_000_000, 6)
    for S in (20_000, 700_000):   # one and four columns per thread
        columns = pinned(np.random.default_rng(S).integers(0, 100_000, S))

        def call(ctx, wait=True):
            out, nnz = torch.full((S + 1 + PAD,), -7, dtype=torch.int64, device="cuda"), ctypes.c_int64(0)
            ctx.check(ctx.lib.gsb_col_slice_count(ctx.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                                  indptr.data_ptr(), 100_000, columns.data_ptr(), S, out.data_ptr(),
                                                  ctypes.byref(nnz) if wait else None), "gsb_col_slice_count")
            assert bool((out[S + 1:] == -7).all())
            return out[:S + 1], nnz.value

        def left_behind(got):   # offsets up to some column, no edges from there on
            offsets = got[0]
            kept = int(np.argmax(np.diff(offsets) < 0)) + 1
            assert np.all(offsets[kept:] == 0) and np.all(np.diff(offsets[:kept]) >= 0)

        run_out(ops, call)
        run_out(ops, lambda ctx: call(ctx, wait=False), left_behind)


@pytest.mark.parametrize("k", [5, 16, 25])
def test_uniform_sampling(ops, k):
    indptr, indices = graph(100_000, 2_000_000, 6)
    columns = pinned(np.random.default_rng(k).integers(0, 100_000, 300_000))
    run_out(ops, lambda ctx: ops.fused_csc_col_slicing_sampling(indptr, indices, columns, k, False, seed=3, ctx=ctx))


@pytest.mark.parametrize("sort", [False, True])
def test_batched_unique(ops, sort):
    rng = np.random.default_rng(9)
    ptr = np.arange(41) * 20_000
    data, d_ptr = dev(rng.integers(0, 50_000, ptr[-1])), dev(ptr)
    run_out(ops, lambda ctx: ops.batch_unique(data, d_ptr, sort=sort, ctx=ctx), tries=50, certain=False)


@pytest.mark.parametrize("path", [1, 2, 3])
def test_batched_relabel_forms(ops, path):
    rng = np.random.default_rng(7)
    sp, ep = np.arange(41) * 500, np.arange(41) * 12_000
    seeds, edges = dev(rng.integers(0, 50_000, sp[-1])), dev(rng.integers(0, 50_000, ep[-1]))
    d_sp, d_ep = dev(sp), dev(ep)

    def call(ctx):
        ctx.set_option("relabel_path", path)
        return ops.batch_csr_relabel(seeds, d_sp, edges, d_ep, ctx=ctx, num_nodes=50_000)[:3]

    run_out(ops, call, tries=50, certain=False)


@pytest.mark.parametrize("path", [0, 1, 3])
def test_queued_hops(ops, path):
    """Three hops without a wait in between: whichever scan is given up, the hops behind it write nothing out of bounds."""
    indptr, indices = graph(100_000, 2_000_000, 5)
    seeds, ptr = pinned(np.arange(16_000)), dev(np.arange(17) * 1000)

    def call(ctx):
        ctx.set_option("relabel_path", path)
        hops = ops.sage_sample_batches(indptr, indices, seeds, ptr, [5, 5, 3], seed=2, ctx=ctx, sync=False)
        return [h["frontier_ptr"] for h in hops]

    run_out(ops, call)


def test_row_slices(ops):
    indptr, indices = graph(100_000, 2_000_000, 6)
    rows = dev(np.random.default_rng(2).permutation(100_000)[:30_000])
    run_out(ops, lambda ctx: ops.csc_row_slicing(indptr, indices, rows, ctx=ctx), tries=50, certain=False)
    cols = ops.csc2coo(indptr, indices)[1]
    run_out(ops, lambda ctx: ops.coo_row_slicing(pinned(indices.cpu().numpy()), cols, rows, ctx=ctx), tries=50)


@pytest.mark.parametrize("presorted", [False, True])
def test_conversion_in_several_launches(ops, presorted):
    E, keys = (4 << 20) + 77, 300_000
    rng = np.random.default_rng(E)
    key, other = rng.integers(0, keys, E), dev(rng.integers(0, 1 << 40, E))
    key = dev(np.sort(key) if presorted else key)
    everything = other.cpu().numpy()

    def left_behind(got):
        indptr, rows, perm = got
        assert indptr[0] == 0 and np.all(indptr[1:] == E) and np.array_equal(rows, everything)
        assert perm is None or np.array_equal(perm, np.arange(E))

    run_out(ops, lambda ctx: ops.coo2csc(other, key, keys, presorted, ctx=ctx), left_behind, tries=20, certain=False)


def test_long_list_sample(ops):
    N, k = 1_000_000, 20_000
    rng = np.random.default_rng(k)
    data, probs = dev(rng.permutation(N)), dev(rng.random(N, dtype=np.float32))

    def left_behind(got):
        assert np.array_equal(got[1], np.arange(k)) and np.array_equal(got[0], data[:k].cpu().numpy())

    run_out(ops, lambda ctx: ops.list_sampling(data, k, False, probs, seed=3, ctx=ctx), left_behind, tries=50, certain=False)
