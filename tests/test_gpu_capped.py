"""Calls under a device allocation budget: what the choice of the sort costs in memory does not refuse a call
that a plainer choice would have room for."""
import pytest

import atc

pytestmark = pytest.mark.gpu


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


def test_small_sorts_take_the_smaller_scratch():
    """preTC of 32 768 pairs took 797 568 bytes with the library's sorts, 846 208 with the own ones."""
    g = atc.rmat_graph(10, 16, 1)
    assert g.shape[0] > 20000

    def call():
        atc.pretc(g, atc.Dir.DEGREE).free()

    assert _least(call, 1 << 24) < 815000
