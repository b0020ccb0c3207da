"""The operators that run as one cooperative launch — COO -> CSC / CSR conversion and list sampling without replacement —
at the sizes where they can go wrong: one item, edges of a warp's and a CTA's share, one, two and three digits, all edges on
one key, the largest call of each and the first beyond it; and the segment kernel's long, short and empty segments."""
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


@pytest.mark.parametrize("E,keys,kind", [
    (1, 1, "uniform"), (31, 40, "uniform"), (1024, 3, "uniform"), (1025, 2048, "uniform"), (2049, 2049, "uniform"),
    (50_000, 1_000_000, "uniform"), (303_104, 5_000_000, "uniform"), (303_105, 77, "uniform"), (200_000, 300_000, "one"),
    (700_001, 100_000, "skewed"), (4 << 20, 1 << 20, "skewed"), ((4 << 20) + 1, 1 << 20, "uniform")])
def test_coo2csc_is_a_stable_sort(ops, E, keys, kind):
    rng = np.random.default_rng(E + keys)
    if kind == "uniform":
        key = rng.integers(0, keys, E)
    elif kind == "one":
        key = np.full(E, keys - 1)
    else:
        key = np.minimum((keys * rng.random(E) ** 4).astype(np.int64), keys - 1)
    key, other = key.astype(np.int64), rng.integers(0, 1 << 40, E).astype(np.int64)
    indptr, out, perm = ops.coo2csc(dev(other), dev(key), keys, False)
    want = np.argsort(key, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), want)
    assert np.array_equal(out.cpu().numpy(), other[want])
    assert np.array_equal(indptr.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(key, minlength=keys))]))


def test_coo2csc_reports_a_key_out_of_range(ops):
    from graph_sampling_b200.cabi import GsbError
    ctx = ops.default_context()
    ops.coo2csc(dev(np.arange(5)), dev(np.array([0, 3, 9, -1, 2])), 4, False)
    with pytest.raises(GsbError) as e:
        ctx.check_device()
    assert e.value.status == -8
    indptr, _, _ = ops.coo2csc(dev(np.arange(3)), dev(np.array([1, 1, 0])), 2, False)
    assert indptr.cpu().tolist() == [0, 1, 3]


@pytest.mark.parametrize("N,k", [(2, 1), (33, 32), (4097, 4096), (5000, 4097), (4096, 7), (1_000_000, 512), (700_001, 4096)])
@pytest.mark.parametrize("weights", [None, "random", "mostly_zero", "equal"])
def test_list_sampling_matches_oracle(ops, oracle, N, k, weights):
    rng = np.random.default_rng(N + k)
    data = rng.permutation(N).astype(np.int64)
    probs = None
    if weights == "random":
        probs = rng.random(N, dtype=np.float32)
    elif weights == "mostly_zero":   # fewer positive weights than picks: the rest are tied at the bottom
        probs = np.zeros(N, np.float32)
        probs[rng.integers(0, N, max(1, k // 2))] = 0.5
    elif weights == "equal":
        probs = np.ones(N, np.float32)
    d, i = ops.list_sampling(dev(data), k, False, None if probs is None else dev(probs), seed=11)
    w_d, w_i = oracle.list_sample(data, probs, k, False, seed=11)
    assert np.array_equal(i.cpu().numpy(), w_i) and np.array_equal(d.cpu().numpy(), w_d)


@pytest.mark.parametrize("lengths", [[1], [0, 0, 5], [2048, 2049, 0, 4, 3, 1], [0] * 5000 + [3, 40, 3000] + [0] * 777, [7] * 9000,
                                     [300_000]])
@pytest.mark.parametrize("permuted", [False, True])
def test_segments_long_short_and_empty(ops, lengths, permuted):
    rng = np.random.default_rng(len(lengths))
    lengths = np.array(lengths)
    indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    data = (rng.random(indptr[-1]) + 0.01).astype(np.float32)
    e_ids = rng.permutation(len(data)).astype(np.int64) if permuted else None
    v = data[e_ids] if permuted else data
    seg = np.repeat(np.arange(len(lengths)), lengths)
    want = np.bincount(seg, v.astype(np.float64) ** 2, len(lengths))
    out = torch.empty(len(lengths), device="cuda")
    d_ids = dev(e_ids) if permuted else None
    got = ops.csc_sum(dev(indptr), d_ids, dev(data), out, 2).cpu().numpy()
    assert np.allclose(got, want, rtol=1e-5, atol=0)
    total = np.bincount(seg, v.astype(np.float64), len(lengths))
    norm = torch.empty(len(data), device="cuda")
    got = ops.csc_normalize(dev(indptr), d_ids, dev(data), norm).cpu().numpy()
    assert np.allclose(got[e_ids] if permuted else got, v / total[seg], rtol=1e-5, atol=0)


def test_segments_share_warps(ops):
    """Several segments per warp and step: ragged ones, empty ones, hubs between them, and more segments too long for a warp
    in one CTA than its list holds."""
    rng = np.random.default_rng(8)
    ragged = rng.integers(0, 300, 40_001) * (rng.random(40_001) < 0.5)
    ragged[[0, 17, 40_000]] = [2049, 5000, 40_000]
    short = rng.integers(0, 12, 300_000)
    crowded = np.zeros(700_000, np.int64)   # a CTA's segments lie 303 104 (normalised) and 606 208 (summed) apart
    for at in (0, 303_104, 606_208):
        crowded[at:at + 256] = 2049
    for lengths in (ragged, short, crowded):
        indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
        E = int(indptr[-1])
        data, seg = (rng.random(E) + 0.01).astype(np.float32), np.repeat(np.arange(len(lengths)), lengths)
        for e_ids in (None, rng.permutation(E)):
            v = data if e_ids is None else data[e_ids]
            total = np.bincount(seg, v.astype(np.float64), len(lengths))
            d_ids, out = None if e_ids is None else dev(e_ids), torch.full((len(lengths),), -1.0, device="cuda")
            got = ops.csc_sum(dev(indptr), d_ids, dev(data), out, 1).cpu().numpy()
            assert np.allclose(got, total, rtol=1e-5, atol=0)
            norm = torch.full((E,), -1.0, device="cuda")
            got = ops.csc_normalize(dev(indptr), d_ids, dev(data), norm).cpu().numpy()
            assert np.allclose(got if e_ids is None else got[e_ids], v / total[seg], rtol=1e-5, atol=0)


def test_segments_beyond_32_bits_of_edges(ops):
    """Offsets within a warp's segments are 32-bit; a step that spans more edges is left to whole CTAs.  Sums of ones, which need
    no data: one segment of 2^30 + 5 edges and one of 2^31 among short ones."""
    import ctypes
    n = 30_000_000
    lengths = torch.full((n,), 3, dtype=torch.int64, device="cuda")
    lengths[12_345], lengths[20_000_001] = (1 << 30) + 5, 1 << 31
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lengths, 0, out=indptr[1:])
    out, ctx = torch.full((n,), -1.0, device="cuda"), ops.default_context()
    ctx.check(ctx.lib.gsb_segment_sum_csc(ctx.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                          indptr.data_ptr(), n, None, None, 1, out.data_ptr()), "gsb_segment_sum_csc")
    assert torch.allclose(out.double(), lengths.double(), rtol=1e-6, atol=0)
