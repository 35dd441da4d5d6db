"""Calls under a device allocation budget: what the choice of the kernel or of the sort costs in memory
does not refuse a call that a plainer choice would have room for."""
import numpy as np
import pytest

import atc
import oracle

pytestmark = pytest.mark.gpu
K = atc.Kernel


@pytest.fixture(autouse=True)
def _lift():
    yield
    atc.set_alloc_budget(None)


def _least(call, hi):
    """The smallest budget (to 1 / 1024) that the call succeeds with."""
    def fits(b):
        atc.set_alloc_budget(b)
        try:
            call()
            return True
        except atc.ATCError as e:
            assert e.status == atc.Status.ERR_OOM, str(e)
            return False
        finally:
            atc.set_alloc_budget(None)
    lo = 0
    assert fits(hi)
    while hi - lo > max(1, hi >> 10):
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid) else (mid, hi)
    return hi


@pytest.mark.parametrize("scale,edge_factor", [(16, 16), (17, 8), (18, 16)])
def test_auto_counts_where_the_hu_style_count_fits(scale, edge_factor):
    g = atc.rmat_graph(scale, edge_factor, 1)
    want = oracle.tc_count(g)
    csr = atc.pretc(g, atc.Dir.ADIRECTION)
    # an item shape keeps the Hu-style count on its work items
    need = _least(lambda: atc.tc(csr, K.HU, tuning={"bisson_slots": 4}), 1 << 28)
    for b in (need, 2 * need, 3 * need):
        atc.set_alloc_budget(b)
        assert atc.tc(csr, K.AUTO)[0] == want, b
        atc.set_alloc_budget(None)
    csr.free()


@pytest.mark.parametrize("mode,before", [(0, 5361664), (1, 5361664)])
def test_batches_take_no_more_than_before(mode, before):
    """Three R-MAT graphs of scale 13: bytes that adding and counting them took before rows items had chunks of
    their own (both modes), to 1 / 1024."""
    csr = atc.pretc(atc.rmat_graph(13, 16, 1), atc.Dir.ADIRECTION)

    def call():
        b = atc.Batch()
        try:
            for _ in range(3):
                b.add(csr)
            return b.run({"group_by_source": mode} if mode else None)
        finally:
            b.free()

    assert _least(call, 1 << 24) <= before * 1025 // 1024
    csr.free()


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("name", ["rmat13", "clique1200", "both"])
def test_rows_items_fit_where_the_groups_did(name, mode):
    """Items of 64 partners at most need no more room than the partner list that graphs counted by rows do not have:
    modes 1 and 2 fit where mode 0 does, on long rows too."""
    u, v = np.triu_indices(1200, 1)
    clique = np.stack([u, v], 1).astype(np.int32)
    graphs = {"rmat13": [atc.rmat_graph(13, 16, 1)], "clique1200": [clique], "both": [atc.rmat_graph(13, 16, 1), clique]}
    csrs = [atc.pretc(g, atc.Dir.ADIRECTION) for g in graphs[name]]
    want = [oracle.tc_count(g) for g in graphs[name]]

    def call(m):
        b = atc.Batch()
        try:
            for c in csrs:
                b.add(c)
            got = b.run({"group_by_source": m} if m else None)
        finally:
            b.free()
        assert [int(x) for x in got[0]] == want
        return got

    assert _least(lambda: call(mode), 1 << 25) <= _least(lambda: call(0), 1 << 25)
    for c in csrs:
        c.free()


def test_batch_modes_in_turn():
    """A change of the mode back and forth keeps its buffers; the counts stay."""
    graphs = [atc.rmat_graph(9 + i % 3, 8, 40 + i) for i in range(6)]
    want = [oracle.tc_count(g) for g in graphs]
    b = atc.Batch()
    for g in graphs:
        c = atc.pretc(g, atc.Dir.ADIRECTION)
        b.add(c)
        c.free()
    for mode in (2, 1, 2, None, 1, 2, None):
        got, _ = b.run({"group_by_source": mode} if mode else None)
        assert [int(x) for x in got] == want, mode
    b.free()


def test_small_sorts_take_the_smaller_scratch():
    """preTC of 32 768 pairs took 797 568 bytes with the library's sorts, 846 208 with the own ones."""
    g = atc.rmat_graph(10, 16, 1)
    assert g.shape[0] > 20000

    def call():
        atc.pretc(g, atc.Dir.DEGREE).free()

    assert _least(call, 1 << 24) < 815000
