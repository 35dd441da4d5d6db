"""k-cliques where few rows are long (split over CTAs), where many are (a warp each), and where every
edge is walked: all against the walk alone and, for complete graphs, the binomials."""
from math import comb

import numpy as np
import pytest

import atc

pytestmark = pytest.mark.gpu


def _planted(n, cliques, size, m, seed):
    rng = np.random.default_rng(seed)
    i, j = np.triu_indices(size, 1)
    e = [rng.integers(0, n, (m, 2))]
    for _ in range(cliques):
        v = rng.permutation(n)[:size]
        e.append(np.stack([v[i], v[j]], 1))
    return np.concatenate(e).astype(np.int32)


@pytest.mark.parametrize("n,cliques,size,m", [(300, 1, 20, 900), (2000, 3, 34, 9000), (20000, 60, 36, 60000),
                                              (60000, 900, 20, 130000), (40000, 2200, 35, 60000),
                                              (30000, 13000, 18, 20000), (5000, 40, 70, 20000)])
@pytest.mark.parametrize("k", [3, 4, 5, 6, 7])
def test_rows_and_walk_agree(n, cliques, size, m, k):
    csr = atc.pretc(_planted(n, cliques, size, m, n + size), atc.Dir.ADIRECTION)
    want = atc.kcl_part(csr, k, 0, 1, dense=False)[0]
    assert atc.kcl(csr, k)[0] == want
    assert sum(atc.kcl_part(csr, k, p, 3)[0] for p in range(3)) == want
    csr.free()


@pytest.mark.parametrize("n", [16, 17, 18, 32, 33, 34, 50, 66])
@pytest.mark.parametrize("k", [3, 4, 5, 6, 7, 8])
def test_complete(n, k):
    i, j = np.triu_indices(n, 1)
    csr = atc.pretc(np.stack([i, j], 1).astype(np.int32), atc.Dir.ID)
    assert atc.kcl(csr, k)[0] == comb(n, k)
    csr.free()


@pytest.mark.parametrize("k", [4, 5, 6])
def test_no_room_for_the_lists(k):
    """Whatever the budget holds, the count is right or refused, by rows or, where only their lists do not
    fit, by the walk."""
    csr = atc.pretc(_planted(40000, 2200, 35, 60000, 3), atc.Dir.ADIRECTION)
    want = atc.kcl(csr, k)[0]
    counted = False
    try:
        for b in range(12, 27):
            for f in (4, 5, 6, 7):
                atc.set_alloc_budget(f << (b - 2))
                try:
                    assert atc.kcl(csr, k)[0] == want
                    counted = True
                except atc.ATCError as e:
                    assert "allocation budget" in str(e)
    finally:
        atc.set_alloc_budget(None)
    assert counted
    csr.free()
