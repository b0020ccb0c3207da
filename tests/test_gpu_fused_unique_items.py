"""The single-launch unique + relabel at the sizes where its items per thread change (1, 2, 3, 4, 5, 6, 8, 12, 16 for one or two CTAs of
512 threads on each of 148 SMs), direct-address and hash table, one minibatch with columns and several, against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
WAVE = 148 * 512   # items of one CTA per SM at one item per thread; two are resident


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("bounded", [False, True])
@pytest.mark.parametrize("n", [2 * WAVE, 3 * WAVE, 3 * WAVE + 1, 6 * WAVE, 6 * WAVE + 1, 8 * WAVE + 1, 10 * WAVE, 10 * WAVE + 1,
                               12 * WAVE + 1, 16 * WAVE + 1, 24 * WAVE + 1])
def test_items_per_thread(oracle, n, bounded):
    from graph_sampling_b200 import ops
    rng = np.random.default_rng(n)
    ids, S = rng.integers(0, n // 2, n), n // 9
    first, second, at = ids[:S], ids[S:], rng.integers(0, S, n - S)
    want, (rows, cols) = oracle.unique_relabel([first, second], [second, first[at]])
    got = ops.graph_relabel(dev(first), dev(second), cols=dev(at), id_bound=n // 2 if bounded else 0)
    for a, b in zip((want, rows, cols), got):
        np.testing.assert_array_equal(a, b.cpu().numpy())
    cut = np.sort(rng.integers(0, n - S, 2))
    sp, ep = np.array([0, S // 3, S // 3, S]), np.concatenate([[0], cut, [n - S]])
    f, fp, rel, _ = (t.cpu().numpy() for t in ops.batch_csr_relabel(dev(first), dev(sp), dev(second), dev(ep),
                                                                  num_nodes=n // 2 if bounded else 0))
    for b in range(3):
        e = second[ep[b]:ep[b + 1]]
        want, (rows,) = oracle.unique_relabel([first[sp[b]:sp[b + 1]], e], [e])
        np.testing.assert_array_equal(want, f[fp[b]:fp[b + 1]])
        np.testing.assert_array_equal(rows, rel[ep[b]:ep[b + 1]])
