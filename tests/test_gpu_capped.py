"""Calls under a device allocation budget: what the choice of the kernel or of the sort costs in memory
does not refuse a call that a plainer choice would have room for."""
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


def test_small_sorts_take_the_smaller_scratch():
    """preTC of 32 768 pairs took 797 568 bytes with the library's sorts, 846 208 with the own ones."""
    g = atc.rmat_graph(10, 16, 1)
    assert g.shape[0] > 20000

    def call():
        atc.pretc(g, atc.Dir.DEGREE).free()

    assert _least(call, 1 << 24) < 815000
