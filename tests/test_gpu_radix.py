"""The key sort under preTC at its edges: around the size where it takes over, whole tiles of 2048
and 8192 keys, the size where the tile states share one buffer, id widths from one pass to eight-bit digits
of every width, and keys that agree in most digits."""
import numpy as np
import pytest

import atc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [4095, 4096, 4097, 6144, 6145, 32769, 73728, (1 << 18), (1 << 18) + 1, (1 << 20), (1 << 20) + 1, (1 << 20) + 8192])
@pytest.mark.parametrize("bits", [3, 8, 9, 17, 22])
@pytest.mark.parametrize("skew", [0, 1])
def test_rows_of_the_sorted_edges(m, bits, skew):
    rng = np.random.default_rng(m + bits)
    e = rng.integers(0, 1 << bits, (m, 2), dtype=np.int64)
    if skew:  # most edges share their source, and a run of them is one edge
        e[: m // 2, 0] = (1 << bits) - 1
        e[m // 4: m // 3] = e[0]
    csr = atc.pretc(e.astype(np.int32), atc.Dir.ID)
    off, cols = csr.to_host()
    lo, hi = e.min(1), e.max(1)
    keys = np.unique(((lo << 32) | hi)[lo != hi])
    src = np.repeat(np.arange(csr.n), np.diff(off))
    got = np.minimum(src, cols) << 32 | np.maximum(src, cols)
    assert csr.m == keys.size and np.array_equal(np.sort(got), keys)
    assert np.all((np.diff(src) > 0) | (np.diff(cols) > 0))  # by source, then ascending
    csr.free()
