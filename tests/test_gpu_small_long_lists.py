"""Small Hu-style counts with a few edges between two long lists, which a block takes together: lists at
the edges of what a lane group keeps (16 elements a lane of 8, 16 or 32), up to thousands of such edges."""
from math import comb

import numpy as np
import pytest

import atc

pytestmark = pytest.mark.gpu
K = atc.Kernel


def _hubs(leaves, hubs):
    """`hubs` hubs over the same leaves, every two of them adjacent; by id the hubs hold the leaves."""
    h = np.arange(leaves, leaves + hubs)
    i, j = np.triu_indices(hubs, 1)
    star = np.stack([np.repeat(h, leaves), np.tile(np.arange(leaves), hubs)], 1)
    return np.concatenate([star, np.stack([h[i], h[j]], 1)]).astype(np.int32)


@pytest.mark.parametrize("leaves,hubs", [(100, 2), (127, 2), (128, 2), (129, 2), (255, 3), (257, 3), (511, 40), (513, 40),
                                         (1025, 12), (5000, 2), (100000, 2), (60000, 3), (900, 80), (300, 200)])
def test_hubs(leaves, hubs):
    csr = atc.pretc(_hubs(leaves, hubs), atc.Dir.ID)
    assert csr.max_outdeg == leaves + hubs - 1
    want = leaves * comb(hubs, 2) + comb(hubs, 3)
    count, stats = atc.tc(csr, K.HU)
    assert count == want
    small = 5.5 * csr.wedges_min + 15 * csr.m < 2 * csr.wedges + 4.7e7 and csr.m <= 1 << 19
    assert (stats.launches == 1) == small
    for parts in (2, 5):
        assert sum(atc.tc_part(csr, p, parts, K.HU)[0] for p in range(parts)) == want
    assert atc.tc(csr, K.AUTO)[0] == want
    csr.free()
