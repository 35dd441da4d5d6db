"""Rows come out ascending from the sort on the source alone (no relabelling), with sources of all
ones, dropped edges and loops; in-degrees and the shorter-list sum from the same passes."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 16, 17, 255, 256, 257, 4096])
@pytest.mark.parametrize("prune", [0, 1])
@pytest.mark.parametrize("dir", list(atc.Dir))
def test_rows_ascend(n, prune, dir):
    rng = np.random.default_rng(n)
    e = rng.integers(0, n, (4 * n, 2))
    # the largest id (2^B - 1 where n is a power of two) has an edge to a leaf and to others
    e = np.concatenate([e, [(n - 1, 0), (0, n - 1), (n - 1, n - 1), (n - 1, n // 2), (n // 2, 0)]]).astype(np.int32)
    csr = atc.pretc(e, dir, tuning={"prune_deg1": prune})
    off, cols = csr.to_host()
    assert off[0] == 0 and off[-1] == csr.m and np.all(np.diff(off) >= 0)
    for u in range(csr.n):
        row = cols[off[u]: off[u + 1]]
        assert np.all(np.diff(row) > 0) and (row.size == 0 or (row[0] >= 0 and row[-1] < csr.n))
    out = np.diff(off)
    src = np.repeat(np.arange(csr.n), out)
    assert csr.wedges == int((np.bincount(cols, minlength=csr.n) * out).sum())
    assert csr.wedges_min == int(np.minimum(out[src], out[cols]).sum())
    assert csr.max_outdeg == (out.max() if csr.n else 0)
    assert atc.tc(csr, atc.Kernel.BISSON)[0] == oracle.tc_count(e)
    simple = {(min(a, b), max(a, b)) for a, b in e.tolist() if a != b}
    if not prune:
        assert csr.m == len(simple)
        assert {(min(a, b), max(a, b)) for a, b in zip(src.tolist(), cols.tolist())} == simple
    csr.free()


def test_negative_ids_and_loops_only():
    with pytest.raises(atc.ATCError, match="negative vertex id -7"):
        atc.pretc(np.array([(3, 4), (-7, 2), (-1, 5)], np.int32))
    csr = atc.pretc(np.array([(3, 3), (5, 5)], np.int32))
    assert csr.m == 0 and csr.n == 6 and atc.tc(csr)[0] == 0
    csr.free()
