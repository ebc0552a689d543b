"""Cell codes stored four at a time: rows of every length modulo 4 that begin
at every offset from a 4-byte boundary, rows shorter than one store, tiles of
128 cells with 1 to 3 cells in the last one, slices of 1 to 9 rows, one to four
levels of a field together, in double and single precision and for row pitches
that TMA can and cannot address.  Counts per cell and images are the oracle's."""
import numpy as np
import pytest

from contour3d_gb300 import _abi
from . import cases

pytestmark = pytest.mark.gpu
NX = [2, 3, 4, 5, 6, 7, 33, 127, 128, 129, 130, 131, 132, 133, 258, 260]


@pytest.mark.parametrize("nx", NX)
@pytest.mark.parametrize("ny,nz", [(4, 5), (9, 4), (10, 3), (18, 4)])
def test_counts(gpu, oracle, nx, ny, nz):
    f = np.random.default_rng(nx * 100 + ny).standard_normal((nz, ny, nx))
    f[nz // 2, ny // 2, nx // 2] = np.nan
    for level in (0.0, -0.8):
        cg, tg = gpu.cell_counts(f, level)
        co, to = oracle.cell_counts(f, level)
        assert tg == to and np.array_equal(cg, co)


@pytest.mark.parametrize("nx", [5, 36, 127, 130, 131, 132, 261])
@pytest.mark.parametrize("levels", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_levels_together(gpu, oracle, nx, levels, dtype):
    torch = pytest.importorskip("torch")
    f = np.random.default_rng(nx + levels).standard_normal((7, 11, nx)).astype(dtype)
    d = torch.from_numpy(f).cuda()
    colors = [(255, 0, 0), (0, 255, 0), (0, 0, 255), (255, 255, 0), (0, 255, 255)]
    values = [0.4 * q - 0.7 for q in range(levels)]
    s = _abi.make_scene(cases.CAM0, cases.CENTRE, 96, 64)
    s.contours = [_abi.Contour(f.astype(np.float64), v, c) for v, c in zip(values, colors)]
    ref = oracle.render(s)
    assert np.array_equal(gpu.render(s), ref)
    out = torch.zeros(64 * 96 * 3, dtype=torch.uint8, device="cuda")
    grids = tuple(_abi.unit_grid(n) for n in (nx, 11, 7))
    rc = gpu.render_device(s, [(d.data_ptr(), int(dtype == "float32"), (nx, 11, 7), grids, v, c)
                               for v, c in zip(values, colors)], out.data_ptr())
    torch.cuda.synchronize()
    assert rc == 0 and np.array_equal(out.cpu().numpy().reshape(64, 96, 3), ref)
