"""btc_trim_memory: the device memory kept from freed handles goes back to the device."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_kept_memory_is_given_back():
    from btc_b200 import BitBSR, graphs as G, trim_memory
    s, d, n = G.rmat_raw_torch(17, 16, 3)
    trim_memory()
    g = BitBSR(s, d, n, 128, orient_degree=True)
    want = g.count()
    g.free()
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    trim_memory(1 << 40)  # everything may stay
    assert torch.cuda.mem_get_info()[0] == kept
    trim_memory()
    assert torch.cuda.mem_get_info()[0] >= kept + (32 << 20)  # the handle held more than that
    g = BitBSR(s, d, n, 128, orient_degree=True)
    trim_memory()  # memory in use stays
    assert g.count() == want
    g.free()
