"""Offsets without allocation at the sizes where their tiles, bit planes and
node ranges end, against the oracle's per-cell counts (integers: exactly)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nz, ny, nx) nodes: one cell; columns of single-cell rows and slices (a node
# range four times the cells); 8,192 cells, so that the end position has a
# tile of its own; tiles that cross row and slice ends; rows just short of and
# just beyond the length whose bits fit in shared memory, and far beyond it
SHAPES = [(2, 2, 2), (9001, 2, 2), (2, 8211, 2), (2, 2, 8193), (17, 17, 33), (9, 7, 1030), (3, 3, 8200), (3, 4, 12400),
          (3, 4, 12500), (3, 3, 40011)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_offsets_at_tile_edges(gpu, oracle, dtype, shape):
    import torch
    rng = np.random.default_rng(sum(shape))
    f = rng.standard_normal(shape).astype(dtype)
    f.flat[::53] = 0.0
    f.flat[1::97] = -0.0
    f.flat[2::211] = np.inf
    f.flat[3::223] = -np.inf
    f.flat[4::227] = np.nan
    dev = torch.from_numpy(f).cuda()
    n = int(np.prod([s - 1 for s in shape]))
    off = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    total = torch.empty(1, dtype=torch.int64, device="cuda")
    sizes = (C.c_size_t * 3)(shape[2], shape[1], shape[0])
    for thr in (0.0, 0.7, -np.inf, np.inf, np.nan):
        off.fill_(-1)
        assert gpu.lib.contour3d_gb300_cell_offsets_noalloc(
            dev.data_ptr(), 0 if dtype is np.float64 else 1, sizes, thr, off.data_ptr(), total.data_ptr(), None) == 0
        counts, tot = oracle.cell_counts(f.astype(np.float64), thr)
        ref = np.concatenate([[0], np.cumsum(counts.reshape(-1), dtype=np.int64)])
        assert int(total[0]) == tot == ref[-1]
        assert np.array_equal(off.cpu().numpy().astype(np.int64), ref), thr
