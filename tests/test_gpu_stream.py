"""The streaming count over the row store: table sizes and the look-ups past the table,
32-bit keys, rows of many chunks, tile ranges, and the tau rule that picks it, each against
the oracle's merge count."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _spread(n, m, clique, seed):
    """m uniform pairs plus a clique of `clique` vertices spread over the whole id range (its
    rows span all column blocks, so look-ups pass any table)."""
    rng = np.random.default_rng(seed)
    e = rng.integers(0, n, (2, m))
    v = np.linspace(0, n - 1, clique).astype(np.int64)
    i, j = np.triu_indices(clique, 1)
    return (np.concatenate([e[0], v[i]]).astype(np.int32),
            np.concatenate([e[1], v[j]]).astype(np.int32))


def _dense_rows(n, dense, seed):
    """`dense` vertices adjacent to most lower ids, the rest sparse: rows of many chunks."""
    rng = np.random.default_rng(seed)
    r, c = [], []
    for u in range(n - dense, n):
        keep = np.nonzero(rng.random(u) < 0.7)[0]
        r.append(np.full(len(keep), u))
        c.append(keep)
    e = rng.integers(0, n, (2, 8 * n))
    return (np.concatenate(r + [e[0]]).astype(np.int32),
            np.concatenate(c + [e[1]]).astype(np.int32))


CASES = {
    # 64-column blocks: at most 256, exactly 256, one more, 512, one more (the 1024-slot table)
    "table_small": lambda: (*_spread(1000, 9000, 20, 1), 1000),
    "table_256": lambda: (*_spread(16384, 160000, 30, 2), 16384),
    "table_257": lambda: (*_spread(16385, 160000, 30, 3), 16385),
    "table_512": lambda: (*_spread(32768, 300000, 40, 4), 32768),
    "table_513": lambda: (*_spread(32769, 300000, 40, 5), 32769),
    # rows that span more than 1,024 column blocks: look-ups past the table
    "past_table": lambda: (*_spread(150001, 1500000, 200, 6), 150001),
    # more than 65,536 column blocks: 32-bit keys
    "wide_keys": lambda: (*_spread(4300001, 2600000, 300, 7), 4300001),
    # rows of more than 32 words, more chunks listed than one walk takes
    "dense_rows": lambda: (*_dense_rows(20000, 200, 8), 20000),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_stream_count_matches_the_oracle(name):
    from btc_b200 import BitBSR
    from oracle import oracle as O
    s, d, n = CASES[name]()
    rp, col, _ = O.lower_csr(s, d, n)
    want = O.tc_merge(rp, col)
    assert want > 0
    ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    for tile_cols in (32, 128):
        for deg in (False, True):
            g = BitBSR(ts, td, n, tile_cols, orient_degree=deg)
            assert g.count() == want, (tile_cols, deg)
            # a lower tau takes the tile kernels, a higher one stays
            if name in ("table_257", "dense_rows"):
                assert g.count(tau=8) == want and g.count(tau=0x7fffffff) == want
                assert g.count() == want
            # tile ranges add up, whatever row blocks they cut
            bounds = g.partition(5)
            parts = [int(g.count_tiles(a, b)) for a, b in zip(bounds[:-1], bounds[1:])]
            assert sum(parts) == want
            t = g.num_tiles
            cut = [0, 1, t // 3, t // 3 + 1, t - 1, t]
            assert sum(int(g.count_tiles(a, b)) for a, b in zip(cut[:-1], cut[1:])) == want
            # an enqueued rebuild of other edges, then of these again
            g.rebuild(td[: len(d) // 2], ts[: len(s) // 2], n, tile_cols, orient_degree=deg,
                      asynchronous=True)
            g.rebuild(ts, td, n, tile_cols, orient_degree=deg, asynchronous=True)
            assert g.count() == want
            g.free()


def test_a_store_that_outgrows_its_first_build():
    """A rebuild with more entries than the first build's store held."""
    from btc_b200 import BitBSR
    from oracle import oracle as O
    n = 9000
    small = _spread(n, 60000, 10, 11)
    large = _spread(n, 400000, 60, 12)
    g = BitBSR(*(torch.from_numpy(x).cuda() for x in small), n, 32)
    for s, d in (small, large, small):
        rp, col, _ = O.lower_csr(s, d, n)
        g.rebuild(torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda(), n, 32)
        assert g.count() == O.tc_merge(rp, col)
    g.free()


def _captured(fn):
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        fn(s)
    return graph


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("deg", [False, True])
def test_a_captured_lower_tau_count_makes_its_own_index(warm, deg):
    """What a lower tau's kernels read beside the tiles is made by the first such count: not
    allocated while capturing, and not taken for made by the handle when only a graph has it
    (deg: grouped edges, no cell pairs from the build)."""
    from btc_b200 import BitBSR
    from oracle import oracle as O
    n = 40000 if deg else 5000
    s, d = _spread(n, (1 << 22) if deg else 150000, 40, 3)
    rp, col, _ = O.lower_csr(s, d, n)
    want = O.tc_merge(rp, col)
    g = BitBSR(torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda(), n, 32, orient_degree=deg)
    if warm:
        assert g.count(tau=4) == want
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    graph = _captured(lambda st: g.count_async(tau=4, stream=st, d_out=out.data_ptr()))
    assert g.count(tau=4) == want  # before any replay
    for _ in range(2):
        out.zero_()
        graph.replay()
        assert int(out.item()) == want
    assert g.count(tau=4) == want
    del graph
    g.free()


def test_a_replayed_batch_rebuild_leaves_no_stale_index():
    """A captured rebuild is replayed on other edges of the same tiles (every id's last bit
    flipped: the same triangles in other rows): a lower tau's count after it finds the index
    of the new edges, whether a count before it made one or not."""
    from btc_b200 import Batch
    from oracle import oracle as O
    gs, want = [], []
    for k in range(3):
        n = 2048 + 512 * k
        s, d = _spread(n, 60000, 30, 20 + k)
        rp, col, _ = O.lower_csr(s, d, n)
        want.append(O.tc_merge(rp, col))
        gs.append((s, d, n))
    src, dst, off, nv = Batch.concat(gs)
    d_src, d_dst = torch.from_numpy(src).cuda(), torch.from_numpy(dst).cuda()
    args = dict(src=d_src, dst=d_dst, offsets=off, num_vertices=nv, tile_cols=32)
    b = Batch(**args)
    assert b.count(tau=4).tolist() == want
    out = torch.zeros(len(gs), dtype=torch.int64, device="cuda")

    def step(st):
        b.rebuild(**args, stream=st, asynchronous=True)
        b.count_async(out.data_ptr(), stream=st)

    graph = _captured(step)
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert out.cpu().tolist() == want
        assert b.count(tau=4).tolist() == want and b.count(tau=4).tolist() == want
        d_src.bitwise_xor_(1)
        d_dst.bitwise_xor_(1)
    del graph
    b.free()


@pytest.mark.parametrize("tile_cols,n", [(32, 600), (32, 3000), (128, 2304)])
def test_dense_graphs_take_the_tensor_cores_and_change_back(tile_cols, n):
    """A dense graph makes no row store; rebuilds of the same geometry that turn sparse and
    dense again are counted by whatever kernel the last tile count predicts."""
    from btc_b200 import Batch, BitBSR, graphs as G
    from oracle import oracle as O
    ks, kd, _ = G.complete(n)
    dense = torch.from_numpy(ks).cuda(), torch.from_numpy(kd).cuda()
    want_d = n * (n - 1) * (n - 2) // 6
    s, d = _spread(n, 40 * n, 20, 5)
    rp, col, _ = O.lower_csr(s, d, n)
    want_s = O.tc_merge(rp, col)
    sparse = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    g = BitBSR(*dense, n, tile_cols)
    assert g.count() == want_d and g.count(tau=0) == want_d
    for asynchronous in (False, True):
        for e, want in ((sparse, want_s), (sparse, want_s), (dense, want_d), (dense, want_d)):
            g.rebuild(*e, n, tile_cols, asynchronous=asynchronous)
            assert g.count() == want and g.count() == want
            b = g.partition(3)
            assert sum(int(g.count_tiles(x, y)) for x, y in zip(b[:-1], b[1:])) == want
    g.free()
    b = Batch([(ks, kd, n), (ks, kd, n)], tile_cols=tile_cols)
    assert b.count().tolist() == [want_d, want_d]
    b.free()
