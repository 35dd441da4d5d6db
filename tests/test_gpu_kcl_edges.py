"""k-cliques by rows of one source where most ids have no edges."""
from math import comb

import numpy as np
import pytest

import atc

pytestmark = pytest.mark.gpu

FILL = 32  # vertices of a filling clique: rows of up to 31


def _complete(n, base=0):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], 1) + base


def _fill(cliques, base):
    i, j = np.triu_indices(FILL, 1)
    b = base + FILL * np.arange(cliques)[:, None]
    return np.stack([(b + i).ravel(), (b + j).ravel()], 1)


@pytest.mark.parametrize("spread", [1, 300, 5000])
@pytest.mark.parametrize("k", [3, 4, 5, 6])
def test_ids_far_apart(spread, k):
    """Most ids without edges: the warps take more sources at a time, or the edges are walked."""
    g = np.concatenate([_complete(40), _fill(700, 40)]).astype(np.int64) * spread
    csr = atc.pretc(g.astype(np.int32), atc.Dir.ID)
    assert atc.kcl(csr, k)[0] == comb(40, k) + 700 * comb(FILL, k)
    csr.free()
