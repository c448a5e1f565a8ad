"""A handle whose last known graph was small or nearly empty, then an enqueued rebuild of a
large one: the count's schedule and its kernel follow the graph that is there."""
from __future__ import annotations

import statistics

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from btc_b200 import BitBSR, graphs as G  # noqa: E402


def _cuda(s, d):
    return torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()


def _count_us(g, out, before):
    """Device time of an enqueued count, each after `before()`."""
    t = []
    for _ in range(5):
        before()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        g.count_async(d_out=out.data_ptr())
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) * 1e3)
    return statistics.median(t)


@pytest.mark.parametrize("tile_cols", [32, 128])
def test_the_grid_does_not_shrink_on_the_last_graphs_tiles(tile_cols):
    """A mesh after three edges on as many vertices, both enqueued after the three edges were
    counted: one CTA took it, 150 to 190 times as slow as the whole GPU.  The bound of
    four is between that and the noise of two runs."""
    s, d, n = G.stencil27(40)
    mesh, few = _cuda(s, d), _cuda(np.array([1, 2, 3], np.int32), np.array([0, 1, 0], np.int32))
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    g = BitBSR(*mesh, n, tile_cols)
    want = g.count()

    def known():
        g.rebuild(*mesh, n, tile_cols)
        g.rebuild(*mesh, n, tile_cols, asynchronous=True)

    def after_few():
        g.rebuild(*few, n, tile_cols)
        assert g.count() == 0
        g.rebuild(*mesh, n, tile_cols, asynchronous=True)

    usual, changed = _count_us(g, out, known), _count_us(g, out, after_few)
    assert int(out.item()) == want and g.count() == want
    assert changed < 4 * usual, (usual, changed)
    g.free()


def test_a_pending_graph_is_counted_from_the_store_its_build_made():
    """A large sparse graph enqueued after a small one looked dense (its edges over the small
    one's tiles): the count went to the tile kernels and allocated their index."""
    def uniform(n, m, seed):
        e = np.random.default_rng(seed).integers(0, n, (2, m)).astype(np.int32)
        return (*_cuda(e[0], e[1]), n)

    large, small = uniform(40000, 600000, 1), uniform(300, 500, 2)
    g = BitBSR(*large, 32)
    want = g.count()

    def cycle(asynchronous):
        g.rebuild(*small, 32)
        g.count()
        g.rebuild(*large, 32, asynchronous=asynchronous)
        got = torch.zeros(1, dtype=torch.int64, device="cuda")
        g.count_async(d_out=got.data_ptr())
        torch.cuda.synchronize()
        assert int(got.item()) == want and g.count() == want
        return g.info().device_bytes

    held = cycle(False)
    assert cycle(True) == held  # the tile kernels' index would have been allocated
    g.free()
