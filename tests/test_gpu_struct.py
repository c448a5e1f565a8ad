"""The struct counts on a caller's own Bit-BSR, which need not be a lower triangle nor square:
sum over the set bits (u, v) of the common columns of rows u and v, a row past the last one
being empty.  Counts are integers: the tolerance is zero."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _tiles(a: np.ndarray, first_col: np.ndarray, tile_cols: int):
    """(indptr, indices, row_indices, blocks) of the 0/1 matrix `a`, whose columns first_col[0],
    first_col[1], ... are given as runs of 128 (a column id is first_col[j // 128] + j % 128)."""
    rows = a.shape[0] // 16
    indptr, indices, row_indices, blocks = [0], [], [], []
    per = 128 // tile_cols
    words = 16 * tile_cols // 32
    for r in range(rows):
        for j, base in enumerate(first_col):
            for p in range(per):
                t = a[16 * r:16 * r + 16, 128 * j + tile_cols * p:128 * j + tile_cols * (p + 1)]
                if not t.any():
                    continue
                indices.append(int(base) // tile_cols + p)
                row_indices.append(r)
                blocks.append(np.packbits(t.astype(np.uint8), axis=1, bitorder="little").view(np.uint32).reshape(words))
        indptr.append(len(indices))
    as_u32 = lambda x: np.asarray(x, np.uint32)
    return as_u32(indptr), as_u32(indices), as_u32(row_indices), np.concatenate(blocks)


def _count(a, first_col, tile_cols):
    """(blocking struct count, the allocation-free tile-wise count)."""
    from btc_b200 import _lib
    L = _lib.lib()
    arrays = [torch.from_numpy(x.view(np.int32)).cuda() for x in _tiles(a, first_col, tile_cols)]
    result = torch.zeros(1, dtype=torch.int64, device="cuda")
    s = _lib.BtcBcsrDevice(indptr=arrays[0].data_ptr(), indices=arrays[1].data_ptr(),
                           row_indices=arrays[2].data_ptr(), blocks=arrays[3].data_ptr(),
                           result=result.data_ptr(), n=a.shape[0], n_row_blocks=a.shape[0] // 16,
                           num_blocks=arrays[1].numel())
    torch.cuda.synchronize()
    assert arrays[1].numel() >= 8 * (a.shape[0] // 16)  # what the streaming count is for
    fn = L.btc_count_triangles_16x128_adaptive if tile_cols == 128 else L.btc_count_triangles_16x32_adaptive
    out = C.c_ulonglong(0)
    assert fn(C.byref(s), 0, None, C.byref(out)) == 0
    assert int(result.item()) == out.value
    assert L.btc_count_bcsr_noalloc(C.byref(s), tile_cols, -1, None, None) == 0
    torch.cuda.synchronize()
    return out.value, int(result.item())


def _want(a, first_col):
    """Plain integers: every set bit (u, v) with v a row, times the rows' common columns."""
    common = (a.astype(np.float64) @ a.astype(np.float64).T).astype(np.int64)  # (exact: below 2^53)
    total = 0
    for j, base in enumerate(first_col):
        for k in range(128):
            v = int(base) + k
            if v < a.shape[0]:
                total += int(common[a[:, 128 * j + k], v].sum())
    return total


def _random(rows, col_runs, p, seed):
    return np.random.default_rng(seed).random((rows, 128 * col_runs)) < p


def _runs(last, k):
    """k runs of 128 columns spread over [0, last], the first rows' columns among them."""
    head = [0, 128, 256, 384]
    tail = np.unique(np.linspace(512, last // 128 * 128, k - len(head)).astype(np.int64) // 128 * 128)
    return np.concatenate([head, tail])


CASES = {
    # a symmetric square matrix: every triangle six times
    "symmetric": lambda: ((lambda m: (m | m.T) & ~np.eye(1536, dtype=bool))(_random(1536, 12, 0.01, 1)),
                          np.arange(12) * 128),
    # an upper triangle with its diagonal
    "upper": lambda: (np.triu(_random(3072, 24, 0.01, 2)), np.arange(24) * 128),
    # slabs of 512 rows of wider matrices: columns past the 256-, 512- and 1,024-slot tables and
    # past 16-bit keys
    "slab_20000": lambda: (_random(512, 60, 0.02, 3), _runs(20000, 60)[:60]),
    "slab_50000": lambda: (_random(512, 60, 0.02, 4), _runs(50000, 60)[:60]),
    "slab_300000": lambda: (_random(512, 60, 0.02, 5), _runs(300000, 60)[:60]),
    "slab_6000000": lambda: (_random(512, 60, 0.02, 6), _runs(6000000, 60)[:60]),
    # rows that end inside a tile's columns: the tile's last columns have no rows
    "ragged": lambda: (_random(1040, 9, 0.03, 7), np.arange(9) * 128),
}


@pytest.mark.parametrize("tile_cols", [32, 128])
@pytest.mark.parametrize("name", sorted(CASES))
def test_struct_count_of_any_matrix(name, tile_cols):
    a, runs = CASES[name]()
    a = a[:, :128 * len(runs)]
    got, tile_wise = _count(a, runs, tile_cols)
    want = _want(a, runs)
    assert want > 0
    assert got == want and tile_wise == want


def test_kernel_time_leaves_allocations_and_waits_out():
    """A wide sparse struct: its per-vertex rows are half a gigabyte that every call allocates
    and frees, over a quarter of the call.  A time that spans them is within 3% of the call's."""
    import statistics
    import time

    import btc_b200
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    n = 3000000
    e = torch.randint(0, n, (2, 2 * n), generator=gen, device="cuda", dtype=torch.int32)
    b = btc_b200.BCSR_16x32_Device()
    btc_b200.convert_coo_to_bcsr_16x32_gpu(b, btc_b200.CooMatrix(e[0].contiguous(), e[1].contiguous(), n))
    kernel, wall = [], []
    for _ in range(7):
        t = time.perf_counter()
        btc_b200.count_triangles_16x32_adaptive(b, kernel_ms=kernel)
        wall.append((time.perf_counter() - t) * 1e3)
    assert 0 < statistics.median(kernel) < 0.9 * statistics.median(wall), (kernel, wall)
    b.free()
