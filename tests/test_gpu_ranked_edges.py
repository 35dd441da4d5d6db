"""The degree-ranked count at the edges of its bitmaps' ranks, on graphs that are counted on it, which each
test checks by the launches of the call."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu
K = atc.Kernel
RANKED = 17  # launches of the ranked copy alone; grouped lists take seven


def _graph(n, core, each, seed):
    """A dense core, leaves on it, and a strip of triangles through all ids, so that every rank has a row."""
    rng = np.random.default_rng(seed)
    ids = rng.permutation(n)
    i, j = np.triu_indices(core, 1)
    hub = ids[:core]
    leaf = np.repeat(ids[core:], each)
    strip = np.arange(n - 2)
    return np.concatenate([np.stack([hub[i], hub[j]], 1), np.stack([leaf, hub[rng.integers(0, core, leaf.size)]], 1),
                           np.stack([strip, strip + 1], 1), np.stack([strip, strip + 2], 1)]).astype(np.int32)


# targets below rank 2^15 - 1, 2^16 - 1 and 2^17 have a kernel each; row bitmaps reach 2^15 rows
@pytest.mark.parametrize("n", [32766, 32767, 32768, 32769, 65534, 65535, 65536, 65537, 131071, 131072, 131073, 200001])
@pytest.mark.parametrize("core,each", [(300, 20), (1000, 8)])
def test_vertex_counts(n, core, each):
    g = _graph(n, core, each, n + core)
    want = oracle.tc_count(g)
    csr = atc.pretc(g, atc.Dir.ADIRECTION)
    for k in (K.BISSON, K.TRICORE, K.FOX):
        count, stats = atc.tc(csr, k)
        assert count == want, k
        assert stats.launches >= RANKED, (k, stats.launches)
        assert atc.tc(csr, k, tuning={"bisson_slots": 4})[0] == want  # the grouped lists
    csr.free()


@pytest.mark.parametrize("leaves,spread", [(20000, 1), (300000, 1), (20000, 4096)])
def test_stars_stay_on_lists(leaves, spread):
    """No wedge to test: the copy's passes would be the whole cost."""
    g = (np.stack([np.zeros(leaves, np.int64), np.arange(1, leaves + 1)], 1) * spread).astype(np.int32)
    csr = atc.pretc(g, atc.Dir.DEGREE)
    for k in (K.BISSON, K.TRICORE, K.FOX, K.AUTO):
        count, stats = atc.tc(csr, k)
        assert count == 0 and stats.launches < RANKED, (k, stats.launches)
    csr.free()
