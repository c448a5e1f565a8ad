"""Tile ranges of graphs whose row blocks differ by far: hubs in natural order, communities, a
clique beside sparse pairs.  The parts add up to the oracle's count, and no part takes longer than
counting everything."""
from __future__ import annotations

import statistics

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from btc_b200 import BitBSR, graphs as G  # noqa: E402
from oracle import oracle as O  # noqa: E402


def _clique_and_pairs(k, n, m, seed):
    rng = np.random.default_rng(seed)
    v = rng.permutation(n)[:k]
    i, j = np.triu_indices(k, 1)
    e = rng.integers(0, n, (2, m))
    return (np.concatenate([v[i], e[0]]).astype(np.int32), np.concatenate([v[j], e[1]]).astype(np.int32), n)


def _communities(n, k, p, seed):
    rng = np.random.default_rng(seed)
    per, m = n // k, int(n // 2 * (n // k - 1) * p)
    c = rng.integers(0, k, m) * per
    e = rng.integers(0, per, (2, m))
    return (c + e[0]).astype(np.int32), (c + e[1]).astype(np.int32), n


GRAPHS = {
    "hubs": lambda: G.rmat_raw_np(16, 8, 7),
    "communities": lambda: _communities(16384, 8, 0.1, 2),
    "clique": lambda: _clique_and_pairs(700, 60000, 300000, 3),
}


def _us(f):
    t = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) * 1e3)
    return statistics.median(t)


@pytest.mark.parametrize("deg", [False, True])
@pytest.mark.parametrize("tile_cols", [32, 128])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_parts_add_up_and_none_takes_longer_than_the_whole(name, tile_cols, deg):
    s, d, n = GRAPHS[name]()
    rp, col, _ = O.lower_csr(s, d, n)
    want = O.tc_merge(rp, col)
    g = BitBSR(torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda(), n, tile_cols, orient_degree=deg)
    assert g.count() == want
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    for parts in (1, 4, 37):
        b = g.partition(parts)
        assert sum(int(g.count_tiles(x, y).item()) for x, y in zip(b[:-1], b[1:])) == want
    whole = _us(lambda: g.count_async(d_out=out.data_ptr()))
    b = g.partition(4)
    for x, y in zip(b[:-1], b[1:]):
        # twice: a part's own launch and cuts, and the noise of two runs
        assert _us(lambda: g.count_tiles(x, y, out=out)) < 2 * whole, (x, y, whole)
    g.free()
