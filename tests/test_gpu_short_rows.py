"""Graphs of short rows, which the row-wise kernel counts faster than the streaming one: batches of
small graphs, uniform pairs of few edges a vertex, a mesh in degree order with narrow tiles.  Counts
against the oracle's through rebuilds, ranges and a captured step; the default tau's time beside
that of one below it, which always takes the row-wise kernel."""
from __future__ import annotations

import statistics

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from btc_b200 import Batch, BitBSR, graphs as G  # noqa: E402
from oracle import oracle as O  # noqa: E402


def _uniform(n, m, seed):
    e = np.random.default_rng(seed).integers(0, n, (2, m)).astype(np.int32)
    return e[0], e[1], n


def _want(g):
    rp, col, _ = O.lower_csr(*g)
    return O.tc_merge(rp, col)


def _us(f):
    t = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) * 1e3)
    return statistics.median(t)


SINGLES = {
    "uniform_4": (lambda: _uniform(131072, 262144, 1), 32, False),
    "uniform_4_degree": (lambda: _uniform(131071, 262144, 2), 128, True),
    "mesh_degree": (lambda: G.stencil27(50), 32, True),
    "uniform_edge_of_rule": (lambda: _uniform(65536, 20 * 16384, 3), 32, False),
}


@pytest.mark.parametrize("name", sorted(SINGLES))
def test_single_graphs(name):
    make, tile_cols, deg = SINGLES[name]
    s, d, n = make()
    want = _want((s, d, n))
    ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    g = BitBSR(ts, td, n, tile_cols, orient_degree=deg)
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert g.count() == want
    # about one time (1.7 to 2.3 when such graphs streamed)
    tau = 63 if tile_cols == 32 else 1023
    default, below = (_us(lambda: g.count_async(d_out=out.data_ptr())),
                      _us(lambda: g.count_async(tau=tau, d_out=out.data_ptr())))
    assert default < 1.4 * below, (default, below)
    b = g.partition(3)
    assert sum(int(g.count_tiles(x, y).item()) for x, y in zip(b[:-1], b[1:])) == want
    for _ in range(3):
        g.rebuild(td, ts, n, tile_cols, orient_degree=deg, asynchronous=True)
        g.count_async(d_out=out.data_ptr())
        torch.cuda.synchronize()
        assert int(out.item()) == want
    # a graph of the same size that streams, and back
    x, y, _ = _uniform(n, 16 * n, 7)
    other = _want((x, y, n))
    g.rebuild(x, y, n, tile_cols, orient_degree=deg)  # (room for its tiles)
    assert g.count() == other
    for edges, count in (((x, y), other), ((s, d), want)) * 2:
        e = [torch.from_numpy(v).cuda() for v in edges]
        g.rebuild(*e, n, tile_cols, orient_degree=deg, asynchronous=True)
        assert g.count() == count and g.count() == count
    g.free()


def _batches():
    rng = np.random.default_rng(5)
    small = [_uniform(int(n), 3 * int(n), 100 + k) for k, n in enumerate(rng.integers(1, 700, 400))]
    wide = [_uniform(n, 2 * n, 200 + k) for k, n in enumerate((40000, 50001, 29999))]
    return {"small": small, "uniform_4": wide}


@pytest.mark.parametrize("tile_cols", [32, 128])
@pytest.mark.parametrize("name", ["small", "uniform_4"])
def test_batches(name, tile_cols):
    graphs = _batches()[name]
    want = [_want(g) for g in graphs]
    src, dst, off, nv = Batch.concat(graphs)
    args = dict(src=torch.from_numpy(src).cuda(), dst=torch.from_numpy(dst).cuda(), offsets=off, num_vertices=nv,
                tile_cols=tile_cols)
    b = Batch(**args)
    assert b.count().tolist() == want
    out = torch.zeros(len(graphs), dtype=torch.int64, device="cuda")
    tau = 63 if tile_cols == 32 else 1023
    default, below = (_us(lambda: b.count_async(out.data_ptr())), _us(lambda: b.count_async(out.data_ptr(), tau=tau)))
    assert default < 1.4 * below, (default, below)
    for _ in range(2):
        b.rebuild(**args, asynchronous=True)
        assert b.count().tolist() == want

    # a captured rebuild and count, whose index lies in buffers the build has reserved
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    fresh = Batch(**args)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=st):
        fresh.rebuild(**args, stream=st, asynchronous=True)
        fresh.count_async(out.data_ptr(), stream=st)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert out.cpu().tolist() == want
    del graph
    fresh.free()
    b.free()


@pytest.mark.parametrize("deg", [False, True])
def test_the_build_makes_the_row_wise_index(deg):
    """A count behind an enqueued rebuild is one kernel: what it reads beside the tiles is made by
    the build (it had been made again by every such count)."""
    from torch.profiler import ProfilerActivity, profile
    n = 600
    s, d, _ = G.complete(n)
    ts, td = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    g = BitBSR(ts, td, n, 32, orient_degree=deg)
    assert g.count() == n * (n - 1) * (n - 2) // 6
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    for _ in range(3):
        g.rebuild(td, ts, n, 32, orient_degree=deg, asynchronous=True)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            g.count_async(d_out=out.data_ptr())
            torch.cuda.synchronize()
        assert int(out.item()) == n * (n - 1) * (n - 2) // 6
        names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
        if not names:
            pytest.skip("no kernel records on this machine")
        assert len(names) == 1 and "k_count_rows" in names[0], names
    g.free()
