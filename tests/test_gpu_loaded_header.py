"""CSR cache files whose header understates the longest row: the rows decide, not the header."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("claimed", [0, 1, 40, 1 << 20])
@pytest.mark.parametrize("host", [False, True])
def test_longest_row_is_the_arrays(tmp_path, claimed, host):
    g = atc.rmat_graph(13, 24, 7)
    csr = atc.pretc(g, atc.Dir.ADIRECTION)
    longest = csr.max_outdeg
    assert longest > 65
    p = tmp_path / "a.csr"
    csr.save(str(p))
    csr.free()
    b = bytearray(p.read_bytes())
    assert np.frombuffer(b, np.int32, 1, 60)[0] == longest  # 8 bytes of name, five int64, three int32
    b[60:64] = np.int32(claimed).tobytes()
    p.write_bytes(bytes(b))
    got = atc.CSR.load(str(p), host_resident=host)
    assert got.max_outdeg == longest
    for k in (3, 4, 5):
        assert atc.kcl(got, k)[0] == oracle.kclique(g, k), k
    for k in (atc.Kernel.BISSON, atc.Kernel.TRICORE, atc.Kernel.HU):
        assert atc.tc(got, k)[0] == oracle.tc_count(g)
    got.free()
