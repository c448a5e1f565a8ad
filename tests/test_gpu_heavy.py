"""The grouped builder where row blocks differ by far: complete graphs around the edge count from
which a row block is built in slices, cliques among sparse pairs, and natural-order lists with a
hub, which are sorted instead.  Arrays against the sort-based builder's, counts against the
oracle's; enqueued rebuilds replay a graph on new contents of the same buffers."""
from __future__ import annotations

import statistics

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from btc_b200 import BitBSR, graphs as G  # noqa: E402
from oracle import oracle as O  # noqa: E402

ARRAYS = ("indptr", "indices", "row_indices", "blocks")


def _same(a, b):
    ha, hb = a.to_host(), b.to_host()
    for k in ARRAYS:
        assert np.array_equal(ha[k], hb[k]), k


def _uniform(n, m, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    e = torch.randint(0, n, (2, m), generator=gen, device="cuda", dtype=torch.int32)
    return e[0].contiguous(), e[1].contiguous()


def _complete(n, m, seed):
    """K_n in random order, made m long by self-loops (which are dropped)."""
    i = torch.triu_indices(n, n, 1, device="cuda").int()
    pad = torch.arange(m - i.shape[1], device="cuda", dtype=torch.int32) % n
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    p = torch.randperm(m, generator=gen, device="cuda")
    return torch.cat([i[0], pad])[p].contiguous(), torch.cat([i[1], pad])[p].contiguous()


def _clique_and_pairs(k, n, m, seed):
    c = _complete(k, k * (k - 1) // 2, seed)
    e = _uniform(n, m, seed + 1)
    ids = torch.randperm(n, device="cuda")[:k].int()
    return torch.cat([ids[c[0].long()], e[0]]), torch.cat([ids[c[1].long()], e[1]])


def _star(n, m, hub, seed):
    """m uniform pairs and one vertex with `hub` neighbours."""
    e = _uniform(n, m, seed)
    s = torch.cat([e[0], torch.full((hub,), n - 1, device="cuda", dtype=torch.int32)])
    d = torch.cat([e[1], torch.arange(hub, device="cuda", dtype=torch.int32)])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    p = torch.randperm(len(s), generator=gen, device="cuda")
    return s[p].contiguous(), d[p].contiguous()


# In K_n every degree is the same, so degree order keeps the ids and row block I holds 256 I + 120
# edges.  A list of m edges has slices from m / 512 + 1 edges a row block on: 8,568 (row block 33)
# is the last without at m = 8,568 * 512, and has them at one edge less.
@pytest.mark.parametrize("m", [8568 * 512, 8568 * 512 - 1])
@pytest.mark.parametrize("tile_cols", [32, 128])
def test_complete_graph_around_the_limit(tile_cols, m):
    n = 2962
    s, d = _complete(n, m, 1)
    a = BitBSR(s, d, n, tile_cols, orient_degree=True)
    b = BitBSR(s, d, n, tile_cols, orient_degree=True, radix=True)
    want = n * (n - 1) * (n - 2) // 6
    for _ in range(3):  # once as built, then against the arrays' capacity
        _same(a, b)
        assert a.count() == want and a.count(tau=0) == want
        a.rebuild(d, s, n, tile_cols, orient_degree=True)
    a.free()
    b.free()


@pytest.mark.parametrize("tile_cols", [32, 128])
@pytest.mark.parametrize("k,n,m", [(2500, 200000, 1300000), (300, 700001, 4300000)])
def test_enqueued_rebuilds_of_new_contents(tile_cols, k, n, m):
    """Degree-ordered lists of 2^22 edges and more: from the second enqueued rebuild on a CUDA graph
    is replayed, on other edges each time (ids flipped in a bit, direction changed)."""
    s, d = _clique_and_pairs(k, n, m, 3)
    assert len(s) >= 1 << 22
    a = BitBSR(s, d, n, tile_cols, orient_degree=True)
    rp, col, _ = O.lower_csr(s.cpu().numpy(), d.cpu().numpy(), n)
    want = O.tc_merge(rp, col)
    assert a.count() == want
    for bit in (1, 4, 64, 2):
        top = n & ~(2 * bit - 1)  # ids below it stay below n
        for t in (s, d):
            t.copy_(torch.where(t < top, t ^ bit, t))
        a.rebuild(s, d, n, tile_cols, orient_degree=True, asynchronous=True)
        out = torch.zeros(1, dtype=torch.int64, device="cuda")
        a.count_async(d_out=out.data_ptr())
        torch.cuda.synchronize()
        assert int(out.item()) == want
        b = BitBSR(s, d, n, tile_cols, orient_degree=True, radix=True)
        _same(a, b)
        b.free()
    a.free()


def _build_us(s, d, n, tile_cols):
    g = BitBSR(s, d, n, tile_cols)
    t = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        g.rebuild(s, d, n, tile_cols)
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) * 1e3)
    return g, statistics.median(t)


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("tile_cols", [0, 32, 128])
def test_a_hub_in_natural_order(tile_cols, host):
    """Too many cells for the bitmap, one row block with a quarter of the edges: not one CTA's work
    (42 ms; a uniform list of the same size takes about one)."""
    n, m, hub = 2000000, 4000000, 1500000
    s, d = _star(n, m, hub, 5)
    if host:
        g = BitBSR(s.cpu().numpy(), d.cpu().numpy(), n, tile_cols)
    else:
        g, us = _build_us(s, d, n, tile_cols)
        even, even_us = _build_us(*_uniform(n, m + hub, 6), n, tile_cols)
        even.free()
        assert us < 8 * even_us, (us, even_us)
    b = BitBSR(s, d, n, g.tile_cols, radix=True)
    _same(g, b)
    assert g.count() == b.count()
    g.free()
    b.free()


def test_a_grid_in_natural_order_is_grouped_as_before():
    """A balanced list the bitmap does not take: the same arrays by the other builder, device and
    host input, open and given widths."""
    s, d, n = G.stencil7(110)
    ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    for tile_cols in (0, 32, 128):
        for src, dst in ((ts, td), (s, d)):
            g = BitBSR(src, dst, n, tile_cols)
            b = BitBSR(ts, td, n, g.tile_cols, radix=True)
            _same(g, b)
            assert g.count() == 0
            g.free()
            b.free()
