"""k-cliques by rows of one source: lengths of N+(u) at the edges of the row kernels, against
the oracle and the warp search (kcl_dense = -1), whole and in parts."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu


def _hub(d, seed, p):
    """A hub (the largest id, so ATC_DIR_ID gives it all d others) over a random graph."""
    rng = np.random.default_rng(seed)
    n_pairs = int(p * d * (d - 1) / 2)
    e = rng.integers(0, d, size=(n_pairs, 2))
    hub = np.stack([np.full(d, d), np.arange(d)], 1)
    return np.concatenate([e[e[:, 0] != e[:, 1]], hub]).astype(np.int32)


@pytest.mark.parametrize("d", [1, 2, 31, 32, 33, 63, 64, 65, 66, 128, 129, 257, 513])
def test_row_lengths(d):
    g = _hub(d, d, min(0.9, 12.0 / max(d, 1) + 0.04))
    csr = atc.pretc(g, atc.Dir.ID)
    assert csr.max_outdeg >= d
    for k in (3, 4, 5, 6, 7, 8, 9, 12):
        want = oracle.kclique(g, k)
        assert atc.kcl(csr, k)[0] == want, k
    csr.free()


@pytest.mark.parametrize("d,k", [(832, 5), (833, 5), (960, 5), (961, 5), (960, 6), (960, 4), (1280, 4), (1281, 4), (1279, 3), (1281, 3), (900, 6)])
def test_longest_rows(d, k):
    g = _hub(d, d, 0.03)
    csr = atc.pretc(g, atc.Dir.ID)
    assert atc.kcl(csr, k)[0] == oracle.kclique(g, k)
    csr.free()


@pytest.mark.parametrize("n", [20, 33, 34, 65, 66, 70, 130])
def test_dense_rows(n):
    """Complete graphs (C0 of every size up to n - 2) and C0 above 64 members."""
    g = np.array([(i, j) for i in range(n) for j in range(i + 1, n)], dtype=np.int32)
    csr = atc.pretc(g, atc.Dir.DEGREE)
    from math import comb
    for k in (3, 4, 5, 6) if n > 70 else (3, 4, 5, 6, 7, 8, 10):
        if comb(n, k) < 1 << 33:
            assert atc.kcl(csr, k)[0] == comb(n, k), k
    csr.free()


@pytest.mark.parametrize("k", [3, 4, 5, 6])
@pytest.mark.parametrize("nparts", [1, 7])
def test_parts_equal_the_warp_search(k, nparts):
    g = atc.rmat_graph(12, 24, 5)
    csr = atc.pretc(g, atc.Dir.ADIRECTION)
    assert csr.max_outdeg > 65
    total = 0
    for p in range(nparts):
        c, rng, _ = atc.kcl_part(csr, k, p, nparts)
        w, rng2, _ = atc.kcl_part(csr, k, p, nparts, dense=False)
        assert rng == rng2 and c == w, (p, c, w)
        total += c
    assert total == atc.kcl(csr, k)[0]
    csr.free()


def test_host_resident_rows():
    g = atc.rmat_graph(11, 16, 2)
    csr = atc.pretc(g, atc.Dir.DEGREE)
    want = [atc.kcl(csr, k)[0] for k in (4, 5)]
    csr.to_host_resident()
    assert [atc.kcl(csr, k)[0] for k in (4, 5)] == want
    csr.free()
