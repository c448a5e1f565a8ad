"""The one-launch builder of small graphs: sizes around its CTAs, its word and edge limits and
the policy's threshold; arrays and counts against the oracle, the width it picks against
btc_select_tile_policy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _uniform(n, m, seed):
    e = np.random.default_rng(seed).integers(0, n, (2, m))
    return e[0].astype(np.int32), e[1].astype(np.int32), n


def _banded(n, m, near, seed):
    """Pairs at most `near` ids apart (local ids: the policy's wide tiles)."""
    rng = np.random.default_rng(seed)
    u = rng.integers(0, n, m)
    v = np.clip(u + rng.integers(-near, near + 1, m), 0, n - 1)
    return u.astype(np.int32), v.astype(np.int32), n


CASES = {
    "one_edge": lambda: (np.array([1], np.int32), np.array([0], np.int32), 2),
    "self_loops": lambda: (np.arange(50, dtype=np.int32), np.arange(50, dtype=np.int32), 50),
    "ragged": lambda: _uniform(257, 2049, 1),           # one edge into a second CTA
    "tiny_dense": lambda: _uniform(33, 5000, 2),         # duplicates, all cells
    "uniform": lambda: _uniform(16384, 131072, 3),
    "banded_small": lambda: _banded(300, 2000, 5, 4),    # n not far above the near distance
    "banded": lambda: _banded(50001, 400000, 20, 5),
    "most_edges": lambda: _uniform(9001, 1 << 19, 6),
    "one_more": lambda: _uniform(9001, (1 << 19) + 1, 7),  # past the limit
    "most_words": lambda: _uniform(131071, 200000, 8),   # 16x32 cell words near 2^20
    "more_words": lambda: _uniform(140000, 200000, 9),   # past the limit
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_small_build_matches_the_oracle(name):
    from btc_b200 import BitBSR, tile_policy
    from oracle import oracle as O
    s, d, n = CASES[name]()
    rp, col, _ = O.lower_csr(s, d, n)
    want = O.tc_merge(rp, col)
    ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    ref = {C: O.bitbsr_build(rp, col, n, C) for C in (32, 128)}

    def check(g, tile_cols):
        h = g.to_host()
        assert h["tile_cols"] == tile_cols
        for k in ("indptr", "indices", "row_indices", "blocks"):
            assert np.array_equal(h[k], ref[tile_cols][k]), (tile_cols, k)
        assert g.count() == want and g.count(tau=0) == want

    pick = tile_policy(ts, td, n)[0]
    for tile_cols in (0, 32, 128):
        width = tile_cols or pick
        g = BitBSR(ts, td, n, tile_cols)
        check(g, width)
        g.rebuild(td, ts, n, tile_cols)
        check(g, width)
        for _ in range(3):  # enqueued; from the second on a captured graph
            g.rebuild(ts, td, n, tile_cols, asynchronous=True)
            g.count_async()
        check(g, width)
        g.rebuild(s, d, n, tile_cols)  # host input
        check(g, width)
        g.free()


def test_small_rebuilds_of_other_shapes():
    """One handle through widths, sizes that outgrow its arrays, an id out of range, and back."""
    from btc_b200 import BitBSR, BtcError
    from btc_b200._lib import BTC_E_RANGE
    from oracle import oracle as O
    g = BitBSR(*(torch.from_numpy(x).cuda() for x in _uniform(300, 500, 11)[:2]), 300)
    for seed, make in enumerate((lambda: _banded(20000, 150000, 9, 12), lambda: _uniform(30000, 500000, 13),
                                 lambda: _uniform(64, 100, 14), lambda: _banded(4000, 30000, 30, 15),
                                 lambda: _uniform(30000, 500000, 16))):
        s, d, n = make()
        rp, col, _ = O.lower_csr(s, d, n)
        ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
        g.rebuild(ts, td, n)
        assert g.count() == O.tc_merge(rp, col)
        bad = ts.clone()
        bad[len(s) // 2] = n
        with pytest.raises(BtcError) as e:
            g.rebuild(bad, td, n)
        assert e.value.status == BTC_E_RANGE
        with pytest.raises(BtcError):
            g.count()
        g.rebuild(ts, td, n, 128)
        assert g.count() == O.tc_merge(rp, col) and g.tile_cols == 128
    g.free()
