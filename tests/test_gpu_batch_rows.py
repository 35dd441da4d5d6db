"""Batches counted by rows: vertex counts at the edges of the bit and tag tables, members that share a
word in numbers around its fields, rows cut into several items, lists of every alignment."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu


def _sharing(n, k, word):
    """Up to k ids below n that fall into one word of a row's tag table."""
    j = np.arange((n - 1) // 1024 + 1)
    ids = j * 1024 + (word - (j + 1) * 661) % 1024
    return ids[ids < n][:k]


def _graph(n, k, seed):
    rng = np.random.default_rng(seed)
    i, j = np.triu_indices(k, 1)
    share = _sharing(n, k, 17)
    i, j = i[j < share.size], j[j < share.size]
    core = rng.permutation(n)[:150]
    a, b = np.triu_indices(150, 1)
    path = np.arange(n - 1)
    return np.concatenate([np.stack([share[i], share[j]], 1), np.stack([core[a], core[b]], 1),
                           np.stack([path, path + 1], 1), rng.integers(0, n, (2 * n, 2)),
                           np.stack([np.repeat(share, 40), rng.integers(0, n, 40 * share.size)], 1)]).astype(np.int32)


@pytest.mark.parametrize("n", [1 << 15, (1 << 15) + 1, 255 << 10, (255 << 10) + 1, 1023 << 10, (1023 << 10) + 1])
@pytest.mark.parametrize("k", [3, 6, 30])
def test_rows(n, k):
    gs = [_graph(n, k, n + k), _graph(700, 9, k), _graph(n // 3, k, k)]
    want = [oracle.tc_count(g) for g in gs]
    b = atc.Batch()
    for g in gs:
        csr = atc.pretc(g, atc.Dir.ID)
        b.add(csr)
        csr.free()
    for t in ({"group_by_source": 1}, {"group_by_source": 2}, {"group_by_source": 1, "bisson_warp_chunk": 33}):
        got, _ = b.run(t)
        assert [int(x) for x in got] == want, t
    b.free()
