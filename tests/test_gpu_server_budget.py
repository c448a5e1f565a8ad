"""The server's HBM budget: what its slots hold stays within it where batches make per-vertex
rows, and a request waits only for memory that is in use."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from btc_b200 import Server  # noqa: E402
from oracle import oracle as O  # noqa: E402


def _uniform(n, m, seed):
    e = np.random.default_rng(seed).integers(0, n, (2, m)).astype(np.int32)
    return e[0], e[1], n


def _want(g):
    rp, col, _ = O.lower_csr(*g)
    return O.tc_merge(rp, col)


def _serve(srv, graphs):
    ids = {srv.submit(*g, borrow=True): k for k, g in enumerate(graphs)}
    got, deadline = {}, time.time() + 60
    while len(got) < len(ids) and time.time() < deadline:
        for r in srv.poll(wait_ms=100):
            got[ids[r["id"]]] = (r["status"], r["count"])
    return [got.get(k) for k in range(len(graphs))]


@pytest.mark.parametrize("tile_cols", [32, 128])
def test_slots_stay_within_the_budget(tile_cols):
    """Batches of sparse random graphs: nearly a tile and a quarter of a chunk of rows an edge."""
    budget = 256 << 20
    graphs = [_uniform(8192, 65536, k) for k in range(60)]
    srv = Server(hbm_budget_bytes=budget, slots=2, tile_cols=tile_cols, solo_edges=1 << 24)
    try:
        assert _serve(srv, graphs) == [(0, _want(g)) for g in graphs]
        st = srv.stats()
        assert 0 < st["peak_device_bytes"] <= budget
        assert st["batches"] < len(graphs)  # (some shared one)
    finally:
        srv.close()


def test_a_request_does_not_wait_for_what_idle_slots_keep():
    """Both slots keep the buffers of small batches; then one request that needs most of the
    budget."""
    budget = 64 << 20
    small = [_uniform(8192, 65536, 100 + k) for k in range(24)]
    large = _uniform(40000, 400000, 7)
    srv = Server(hbm_budget_bytes=budget, slots=2, max_batch_graphs=4, solo_edges=1 << 24)
    try:
        assert _serve(srv, small) == [(0, _want(g)) for g in small]
        assert _serve(srv, [large]) == [(0, _want(large))]
        assert _serve(srv, small[:5]) == [(0, _want(g)) for g in small[:5]]
    finally:
        srv.close()
