"""Small Hu-style counts of one CSR that overlap on several streams, and the count after them."""
import threading

import pytest
import torch

import atc
import oracle

pytestmark = pytest.mark.gpu
K = atc.Kernel


@pytest.mark.parametrize("scale", [8, 10, 14])
def test_overlapping_counts_share_nothing(scale):
    g = atc.rmat_graph(scale, 16, scale)
    want = oracle.tc_count(g)
    csr = atc.pretc(g, atc.Dir.DEGREE)
    count, stats = atc.tc(csr, K.HU)
    assert count == want and stats.launches == 1  # the small kernel
    streams = [torch.cuda.Stream() for _ in range(4)]
    start = threading.Barrier(len(streams))
    got = [[] for _ in streams]

    def work(i):
        start.wait()
        for _ in range(200):
            got[i].append(atc.tc(csr, K.HU, stream=streams[i].cuda_stream)[0])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(streams))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [sorted(set(x)) for x in got] == [[want]] * len(streams)
    for _ in range(3):  # a later count alone
        assert atc.tc(csr, K.HU)[0] == want
    csr.free()
