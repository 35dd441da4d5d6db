"""Edges tested as bitmap words (long prefixes before targets of low rank): row counts and ranks at
the edges of the 128-bit pieces, sources beyond the bitmap rows, and no room for the bitmaps."""
from math import comb

import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu
K = atc.Kernel


@pytest.mark.parametrize("n", [183, 255, 256, 257, 383, 384, 385, 641])
def test_pieces(n):
    """A complete graph less one vertex's edges to every fifth other, and a pendant path."""
    i, j = np.triu_indices(n, 1)
    keep = ~((i == n // 2) & (j % 5 == 0) | (j == n // 2) & (i % 5 == 0))
    g = np.stack([i[keep], j[keep]], 1)
    g = np.concatenate([g, [(n - 1, n), (n, n + 1)]]).astype(np.int32)
    d = n - 1 - int(np.sum(np.arange(n)[np.arange(n) != n // 2] % 5 == 0))
    csr = atc.pretc(g, atc.Dir.ID)
    assert atc.tc(csr, K.BISSON)[0] == comb(n - 1, 3) + comb(d, 2)
    csr.free()


def _core_and_leaves(n, core, each, seed):
    rng = np.random.default_rng(seed)
    ids = rng.permutation(n)
    i, j = np.triu_indices(core, 1)
    hub = ids[:core]
    leaf = np.repeat(ids[core:], each)
    to = hub[rng.integers(0, core, leaf.size)]
    return np.concatenate([np.stack([hub[i], hub[j]], 1), np.stack([leaf, to], 1),
                           rng.integers(0, n, (2 * n, 2))]).astype(np.int32)


@pytest.mark.parametrize("n,core,each", [(700, 150, 40), (20000, 600, 40), (40000, 257, 48), (70000, 1300, 20)])
def test_sources_beyond_the_rows(n, core, each):
    g = _core_and_leaves(n, core, each, n)
    want = oracle.tc_count(g)
    for d in (atc.Dir.ID, atc.Dir.ADIRECTION):
        csr = atc.pretc(g, d)
        for k in (K.BISSON, K.AUTO):
            assert atc.tc(csr, k)[0] == want, (d, k)
        csr.free()


def test_no_room_for_the_bitmaps():
    g = _core_and_leaves(20000, 600, 40, 5)
    want = oracle.tc_count(g)
    csr = atc.pretc(g, atc.Dir.ADIRECTION)
    try:
        # the bitmaps take up to 4 bytes an edge of a copy of 12 and more: some of these budgets
        # hold the one and not the other
        for b in range(8, 32):
            atc.set_alloc_budget(b * csr.m + 80 * csr.n)
            assert atc.tc(csr, K.BISSON)[0] == want, b
    finally:
        atc.set_alloc_budget(None)
    csr.free()
