"""Descending-degree order: the degree count on both sides of the list length that picks its
table, with more vertices than any table holds, hubs, duplicates and self-loops; the arrays
against the oracle's on ids relabelled by numpy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _edges(n, m, hubs, seed):
    """m uniform pairs, a third of them with one end among `hubs` ids."""
    rng = np.random.default_rng(seed)
    e = rng.integers(0, n, (2, m))
    e[0, : m // 3] = rng.integers(0, hubs, m // 3) * (n // hubs)
    e[1, m // 2: m // 2 + 7] = e[0, m // 2: m // 2 + 7]  # self-loops count nothing
    return e[0].astype(np.int32), e[1].astype(np.int32)


def _by_degree(s, d, n):
    keep = s != d
    deg = np.bincount(s[keep], minlength=n) + np.bincount(d[keep], minlength=n)
    order = np.lexsort((np.arange(n), -deg))  # most edges first, ties by id
    rank = np.empty(n, np.int64)
    rank[order] = np.arange(n)
    return rank[s].astype(np.int32), rank[d].astype(np.int32)


@pytest.mark.parametrize("n,m,hubs", [(2, 1, 1), (300, 255, 3), (300, 257, 3), (5000, (1 << 16) - 1, 7),
                                      (5000, 1 << 16, 7), (90001, (1 << 16) + 1, 40), (90001, 700001, 1)])
def test_degree_order_matches_numpy(n, m, hubs):
    from btc_b200 import BitBSR
    from oracle import oracle as O
    s, d = _edges(n, m, hubs, n + m)
    rs, rd = _by_degree(s, d, n)
    rp, col, _ = O.lower_csr(rs, rd, n)
    for tile_cols in (32, 128):
        ref = O.bitbsr_build(rp, col, n, tile_cols)
        g = BitBSR(torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda(), n, tile_cols, orient_degree=True)
        h = g.to_host()
        for k in ("indptr", "indices", "row_indices", "blocks"):
            assert np.array_equal(h[k], ref[k]), (tile_cols, k)
        assert g.count() == O.tc_merge(rp, col)
        g.free()
