"""The persistent peel loop: lists at the edges of its pieces, levels that admit nobody, isolated
vertices, against the oracle's serial peels."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu


def _star(d):
    return np.stack([np.zeros(d, np.int32), np.arange(1, d + 1, dtype=np.int32)], 1)


def _clique(n, base):
    i, j = np.triu_indices(n, 1)
    return (np.stack([i, j], 1) + base).astype(np.int32)


CASES = {
    **{"star%d" % d: _star(d) for d in (1, 31, 32, 33, 255, 256, 257, 513, 5000)},
    # the dense cores lie many outer steps above the paths: whole runs of steps admit nobody
    "cliques+path": np.concatenate([_clique(300, 0), _clique(700, 300), np.stack(
        [np.arange(1000, 9000), np.arange(1001, 9001)], 1).astype(np.int32)]),
    # ids without edges between and above the others
    "isolated": np.array([(3, 900), (900, 901), (901, 3), (5000, 5001), (7000, 7000)], np.int32),
    "one edge": np.array([(0, 1)], np.int32),
    **{"rmat%d-%d" % (s, ef): atc.gen_rmat(s, ef, s) for s, ef in ((8, 4), (11, 64), (15, 3), (17, 30))},
}


@pytest.mark.parametrize("name", list(CASES))
def test_priorities_and_core_numbers(name):
    g = CASES[name]
    got, prio = atc.adirection(g, want_prio=True)
    want, wprio = oracle.adirection(g, want_prio=True)
    assert np.array_equal(got, want)
    assert np.array_equal(prio, wprio)
    e = (g[:, 0].astype(np.uint64) << np.uint64(32)) | g[:, 1].astype(np.uint64)
    _, core = atc.kcore_direction(e, want_core=True)
    assert np.array_equal(core, oracle.core_numbers(g))
