"""The degree-ranked count (ATC_KERNEL_BISSON on whole CSRs built by preTC): row lengths at the
edges of its row sorts, vertex counts at the edges of its bitmaps, its fallbacks."""
from math import comb

import numpy as np
import pytest
import torch

import atc
import oracle

pytestmark = pytest.mark.gpu
K = atc.Kernel


def _complete(n):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], 1).astype(np.int32)


def _device(pairs, d=atc.Dir.DEGREE):
    torch.cuda.synchronize()
    return atc.pretc_device(pairs.data_ptr(), pairs.shape[0], d)


@pytest.mark.parametrize("n", [3, 4, 32, 33, 34, 64, 65, 66, 128, 130, 257, 258, 513, 514, 1024, 1025, 1026, 1500, 2049])
def test_row_lengths(n):
    csr = atc.pretc(_complete(n), atc.Dir.ID)
    assert atc.tc(csr, K.BISSON)[0] == comb(n, 3)
    csr.free()


@pytest.mark.parametrize("n", [32767, 32768, 32769, 40000, 524287, 524289, 700001])
def test_vertex_counts(n):
    """A triangle strip (every rank has a row) plus a random dense core on scattered ids."""
    rng = np.random.default_rng(n)
    i = np.arange(n - 2)
    core = rng.permutation(n)[:400]
    e = core[rng.integers(0, 400, (30000, 2))]
    g = np.concatenate([np.stack([i, i + 1], 1), np.stack([i, i + 2], 1), e]).astype(np.int32)
    want = oracle.tc_count(g)
    for d in (atc.Dir.ID, atc.Dir.ADIRECTION):
        csr = atc.pretc(g, d)
        for k in (K.BISSON, K.AUTO, K.HU):
            assert atc.tc(csr, k)[0] == want, (d, k)
        csr.free()


@pytest.mark.parametrize("dir", list(atc.Dir))
@pytest.mark.parametrize("tuning", [None, {"prune_deg1": 1}])
def test_equals_the_grouped_lists(dir, tuning):
    """Every orientation; an item shape in the tuning keeps the grouped-list count."""
    g = atc.rmat_graph(14, 20, 9)
    csr = atc.pretc(g, dir, tuning=tuning)
    want = oracle.tc_count(g)
    assert atc.tc(csr, K.BISSON)[0] == want
    assert atc.tc(csr, K.BISSON, tuning={"bisson_slots": 4})[0] == want
    parts = [atc.tc_part(csr, p, 3, K.BISSON)[0] for p in range(3)]
    assert sum(parts) == want
    csr.free()


@pytest.mark.parametrize("n", [3, 17, 33, 34, 65, 129, 181, 183, 257, 258, 600, 1100, 2100])
@pytest.mark.parametrize("kernel", [K.TRICORE, K.FOX])
def test_searched_families(n, kernel):
    """Complete graphs (lists of every length up to n - 1) with their ids scattered over 2^20, so
    that the part tables are sparse; from 16384 edges on the ranked copy, otherwise whole lists."""
    ids = np.random.default_rng(n).choice(1 << 20, n, replace=False).astype(np.int32)
    csr = atc.pretc(ids[_complete(n)], atc.Dir.DEGREE)
    assert atc.tc(csr, kernel)[0] == comb(n, 3)
    assert atc.tc(csr, kernel, tuning={"bisson_slots": 4})[0] == comb(n, 3)
    csr.free()


def test_loaded_rows_that_are_no_orientation(tmp_path):
    """A cache file may hold any sorted rows: its count stays the sum over its rows' edges."""
    n = 50
    adj = [[j for j in range(n) if j != i] for i in range(n)]
    off = np.concatenate([[0], np.cumsum([len(a) for a in adj])]).astype(np.int64)
    cols = np.concatenate(adj).astype(np.int32)
    p = tmp_path / "sym.csr"
    with open(p, "wb") as f:
        f.write(b"ATCCSR01")
        f.write(np.array([n, len(cols), n, 0, 0], dtype=np.int64).tobytes())
        f.write(np.array([0, 0, 0, n - 1], dtype=np.int32).tobytes())
        f.write(off.tobytes())
        f.write(cols.tobytes())
    csr = atc.CSR.load(str(p))
    for k in (K.HU, K.BISSON, K.FOX, K.TRICORE):
        assert atc.tc(csr, k)[0] == n * (n - 1) * (n - 2)
    csr.free()


def test_no_room_for_the_copy():
    g = atc.rmat_graph(12, 16, 3)
    csr = atc.pretc(g, atc.Dir.ADIRECTION)
    want = oracle.tc_count(g)
    try:
        # the grouped lists take 4 bytes an edge and about 70 a vertex, the ranked copy 12 and more
        # than 50: with 12 edges a vertex only the first fit
        assert csr.m > 8 * csr.n
        atc.set_alloc_budget(4 * csr.m + 80 * csr.n)
        assert atc.tc(csr, K.BISSON)[0] == want
    finally:
        atc.set_alloc_budget(None)
    csr.free()


def test_rows_too_long_for_the_sort():
    n = 16400
    i, j = torch.triu_indices(n, n, 1, device="cuda")
    csr = _device(torch.stack([i, j], 1).to(torch.int32).contiguous())
    assert atc.tc(csr, K.BISSON)[0] == comb(n, 3)
    csr.free()


def test_long_rows_beyond_the_bitmaps():
    """Targets of rank 2^19 and above with more than 512 successors."""
    import ctypes
    n, degree = 560000, 1150.0
    cap = int(n * degree * 0.6)
    out = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
    cnt = ctypes.c_uint64(0)
    assert atc.lib().atc_gen_rgg_device(n, degree, 3, out.data_ptr(), cap, ctypes.byref(cnt), None) == 0
    csr = _device(out[: cnt.value])
    assert csr.max_outdeg > 512
    assert atc.tc(csr, K.BISSON)[0] == atc.tc(csr, K.HU)[0]
    csr.free()


@pytest.mark.parametrize("n", [3, 9, 20, 33, 70, 200, 300])
def test_small_counts(n):
    """The small Hu-style kernel (8, 16 and 32 lanes an edge by the mean list), on one CSR several
    times over (its accumulator is left at zero), whole and in parts, beside the item kernels."""
    rng = np.random.default_rng(n)
    e = rng.integers(0, 4 * n, (6 * n, 2))
    hub = np.stack([np.zeros(3 * n, np.int64), np.arange(1, 3 * n + 1)], 1)
    g = np.concatenate([_complete(n), e, hub]).astype(np.int32)
    want = oracle.tc_count(g)
    for d in (atc.Dir.ID, atc.Dir.DEGREE):
        csr = atc.pretc(g, d)
        for _ in range(3):
            assert atc.tc(csr, K.HU)[0] == want
        assert sum(atc.tc_part(csr, p, 5, K.HU)[0] for p in range(5)) == want
        assert atc.tc(csr, K.BISSON)[0] == want
        assert atc.tc(csr, K.HU, tuning={"bisson_slots": 2})[0] == want
        assert atc.tc(csr, K.AUTO)[0] == want
        csr.free()


@pytest.mark.parametrize("cliques,size", [(20000, 9), (4000, 50), (1400, 97), (300, 260), (110, 700)])
def test_targets_of_large_rank(cliques, size):
    """Disjoint cliques on scattered ids, joined in a path: rows of every alignment, members that share
    a bit of the filter, more of them in one item than a stack holds, mean lists on both sides of
    the lane and CTA rules."""
    n = cliques * size
    assert n > 1 << 16
    i, j = torch.triu_indices(size, size, 1, device="cuda")
    first = torch.arange(cliques, device="cuda") * size
    e = torch.stack([(first[:, None] + i).flatten(), (first[:, None] + j).flatten()], 1)
    link = torch.stack([first[:-1], first[1:] + size - 1], 1)  # closes no triangle
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(size)).cuda()
    pairs = perm[torch.cat([e, link])].to(torch.int32).contiguous()
    csr = _device(pairs, atc.Dir.ADIRECTION)
    assert atc.tc(csr, K.BISSON)[0] == cliques * comb(size, 3)
    csr.free()
