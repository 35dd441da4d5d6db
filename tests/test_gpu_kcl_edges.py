"""The k-clique row kernels at the edges of their row lengths.  Disjoint cliques of 32 beside the rows under
test make the graph one that is counted by rows, which each test checks by the launches of the call."""
from math import comb

import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu

FILL = 32  # vertices of a filling clique: rows of up to 31


def _complete(n, base=0):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], 1) + base


def _fill(cliques, base):
    i, j = np.triu_indices(FILL, 1)
    b = base + FILL * np.arange(cliques)[:, None]
    return np.stack([(b + i).ravel(), (b + j).ravel()], 1)


def _by_rows(csr, k, want):
    count, stats = atc.kcl(csr, k)
    assert count == want, k
    # the walk is one launch, from k = 5 on with its dense kernel for lists above 64 two; rows of more than 32
    # members (16 from k = 6 on) are at least one more
    least = 1 + (k >= 5 and csr.max_outdeg > 64)
    assert stats.launches > least or csr.max_outdeg <= (16 if k >= 6 else 32), (k, stats.launches)


# 505 filling cliques have 7575 rows of 17..31 members, few enough to be split over CTAs from k = 6 on;
# 2000 have 30 000, a warp each, and edges enough for rows at k = 3
@pytest.mark.parametrize("cliques", [505, 2000])
@pytest.mark.parametrize("n", [20, 33, 34, 35, 65, 66, 67, 129, 130, 131, 132, 193, 194, 385, 386, 514, 515, 516, 961, 962])
def test_complete_rows(n, cliques):
    """Complete graphs: rows and candidate sets of every length up to n - 1 and n - 2."""
    csr = atc.pretc(np.concatenate([_complete(n), _fill(cliques, n)]).astype(np.int32), atc.Dir.ID)
    assert csr.max_outdeg == max(n, FILL) - 1
    for k in (3, 4, 5, 6, 7) if n <= 67 else (3, 4, 5, 6) if n <= 132 else (3, 4, 5) if n <= 516 else (3, 4):
        if k > 3 or cliques == 2000:
            _by_rows(csr, k, comb(n, k) + cliques * comb(FILL, k))
    csr.free()


@pytest.mark.parametrize("n", [13, 17, 18, 33, 34, 40])
def test_deep_searches(n):
    """From k = 8 on rows are for graphs of few wedges: cliques of 12 for filling."""
    i, j = np.triu_indices(12, 1)
    b = n + 12 * np.arange(5000)[:, None]
    fill = np.stack([(b + i).ravel(), (b + j).ravel()], 1)
    csr = atc.pretc(np.concatenate([_complete(n), fill]).astype(np.int32), atc.Dir.ID)
    for k in (8, 9, 10, 12):
        _by_rows(csr, k, comb(n, k) + 5000 * comb(12, k))
    csr.free()


@pytest.mark.parametrize("d", [31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 192, 193, 257, 384, 385, 513, 832, 833, 960, 961])
def test_sparse_rows(d):
    """A source of d members over a random graph of them."""
    rng = np.random.default_rng(d)
    p = min(0.9, 12.0 / d + 0.04)
    e = rng.integers(0, d, size=(int(p * d * (d - 1) / 2), 2))
    hub = np.stack([np.full(d, d), np.arange(d)], 1)
    g = np.concatenate([e[e[:, 0] != e[:, 1]], hub]).astype(np.int32)
    csr = atc.pretc(np.concatenate([g, _fill(505, d + 1)]).astype(np.int32), atc.Dir.ID)
    for k in (4, 5, 6, 7):
        want = oracle.kclique(g, k) + 505 * comb(FILL, k)
        _by_rows(csr, k, want)
        assert sum(atc.kcl_part(csr, k, q, 3)[0] for q in range(3)) == want, k
    csr.free()


@pytest.mark.parametrize("spread", [1, 300, 5000])
@pytest.mark.parametrize("k", [3, 4, 5, 6])
def test_ids_far_apart(spread, k):
    """Most ids without edges: the warps take more sources at a time, or the edges are walked."""
    g = np.concatenate([_complete(40), _fill(700, 40)]).astype(np.int64) * spread
    csr = atc.pretc(g.astype(np.int32), atc.Dir.ID)
    assert atc.kcl(csr, k)[0] == comb(40, k) + 700 * comb(FILL, k)
    csr.free()
