"""The grouped builder (large edge lists, and sparse ones on many vertices): its arrays equal
the oracle's word for word at both widths, its counts the oracle's merge count."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _uniform(n, m, seed):
    e = np.random.default_rng(seed).integers(0, n, (2, m))
    return e[0].astype(np.int32), e[1].astype(np.int32), n


def _hubs(n, hubs, m, seed):
    """`hubs` neighbouring high rows with many lower neighbours (a row block of far more tiles
    than are built at once), uniform pairs, duplicates and self-loops."""
    rng = np.random.default_rng(seed)
    h = np.repeat(np.arange(n - hubs, n), m // hubs)
    c = rng.integers(0, n, len(h))
    e = rng.integers(0, n, (2, m // 4))
    d = rng.integers(0, n, 1000)
    s = np.concatenate([h, e[0], e[0][:500], d, c[:3000]])
    t = np.concatenate([c, e[1], e[1][:500], d, c[1:3001]])
    return s.astype(np.int32), t.astype(np.int32), n


def _dense(n, seed):
    """K_n with some pairs listed twice, in random order."""
    i, j = np.triu_indices(n, 1)
    p = np.random.default_rng(seed).permutation(len(i))
    i, j = i[p], j[p]
    return (np.concatenate([i, j[:1000]]).astype(np.int32),
            np.concatenate([j, i[:1000]]).astype(np.int32), n)


CASES = {
    # too many cells for the bitmap: any number of edges
    "empty": lambda: _uniform(1600000, 0, 1),
    "one": lambda: (np.array([1599999], np.int32), np.array([0], np.int32), 1600000),
    "sparse": lambda: _uniform(1600001, 300000, 2),
    "tile_of_edges": lambda: _uniform(1599991, 8192, 3),
    "tile_and_one": lambda: _uniform(1599991, 8193, 4),
    "hubs": lambda: _hubs(1600003, 20, 1200000, 5),
    # more edges than the bitmap builder is used for
    "uniform_large": lambda: _uniform(40000, 4500000, 6),
    "dense": lambda: _dense(3001, 7),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_grouped_build_matches_the_oracle(name):
    from btc_b200 import BitBSR
    from oracle import oracle as O
    s, d, n = CASES[name]()
    rp, col, _ = O.lower_csr(s, d, n)
    want = O.tc_merge(rp, col)
    ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    for tile_cols in (32, 128):
        ref = O.bitbsr_build(rp, col, n, tile_cols)
        g = BitBSR(ts, td, n, tile_cols)

        def check():
            h = g.to_host()
            for k in ("indptr", "indices", "row_indices", "blocks"):
                assert np.array_equal(h[k], ref[k]), (tile_cols, k)
            assert g.count() == want and g.count(tau=4) == want

        check()
        # again against the arrays' capacity, waiting and enqueued (a captured graph from the
        # second identical one on)
        g.rebuild(td, ts, n, tile_cols)
        check()
        for _ in range(3):
            g.rebuild(ts, td, n, tile_cols, asynchronous=True)
            assert g.count() == want
        check()
        # in degree order the tiles differ and the count does not
        g.rebuild(ts, td, n, tile_cols, orient_degree=True)
        assert g.count() == want
        g.free()


def test_grouped_build_rejects_ids_out_of_range():
    from btc_b200 import BitBSR, BtcError
    from btc_b200._lib import BTC_E_RANGE
    s, d, n = _uniform(1600001, 20000, 9)
    g = BitBSR(torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda(), n, 128)
    for bad in (-1, n, 0x7fffffff):
        x = s.copy()
        x[777] = bad
        with pytest.raises(BtcError) as e:
            g.rebuild(torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda(), n, 128)
        assert e.value.status == BTC_E_RANGE
    g.free()


def test_degree_order_and_the_bitmap_builder_agree():
    """A degree-ordered list long enough to be grouped, against the sort-based builder."""
    from btc_b200 import BitBSR, graphs as G
    s, d, n = G.rmat_raw_torch(18, 17, 3)
    for tile_cols in (32, 128):
        a = BitBSR(s, d, n, tile_cols, orient_degree=True)
        b = BitBSR(s, d, n, tile_cols, orient_degree=True, radix=True)
        ha, hb = a.to_host(), b.to_host()
        for k in ("indptr", "indices", "row_indices", "blocks"):
            assert np.array_equal(ha[k], hb[k]), (tile_cols, k)
        assert a.count() == b.count() == a.count(tau=64)
        a.free()
        b.free()
