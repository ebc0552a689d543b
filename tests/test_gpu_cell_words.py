"""The scan's word per crossed cell (offset of its first edge, its edges,
whether it is rendered) where it can go wrong: grids whose cells end before, at
and after the end of a scan segment of 8192 cells, rows and slices that
straddle one, fields with no inner cell, crossings in every cell, slabs that
begin inside the field.  Images are the oracle's."""
import numpy as np
import pytest

from contour3d_gb300 import _abi
from . import cases

pytestmark = pytest.mark.gpu

# (nz, ny, nx) in points; cells per grid in the comment
SHAPES = [
    (2, 2, 2),      # 1: nothing is rendered
    (3, 9, 4),      # 48: no inner cell along z
    (4, 4, 4),      # 27: one inner cell
    (17, 17, 33),   # 8192: one segment
    (2, 92, 91),    # 8190, one slice
    (17, 33, 33),   # 16384: two segments
    (4, 51, 56),    # 8250: the last segment holds 58 cells
    (12, 32, 25),   # 8184
    (30, 7, 300),   # rows of 299 cells
    (9, 200, 5),
]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("kind", ["noise", "plane"])
def test_words_at_segment_edges(gpu, oracle, shape, kind):
    rng = np.random.default_rng(sum(shape))
    f = rng.standard_normal(shape)
    if kind == "plane":  # few crossed cells: most segments' groups hold none
        f = np.broadcast_to(np.arange(shape[1], dtype=np.float64)[None, :, None] - 0.47 * shape[1], shape) + 1e-3 * f
    s = _abi.make_scene(cases.CAM0, cases.CENTRE, 90, 70)
    s.contours = [_abi.Contour(f, 0.1, (255, 0, 0)), _abi.Contour(f, -0.3, (0, 0, 255))]
    ref = oracle.render(s)
    assert np.array_equal(gpu.render(s), ref)
    assert np.array_equal(gpu.render(s), ref)  # unsynchronised


@pytest.mark.parametrize("slices", [2, 3, 7])
def test_words_of_slabs(gpu, oracle, slices):
    rng = np.random.default_rng(slices)
    f = rng.standard_normal((23, 31, 29))
    s = _abi.make_scene(cases.CAM0, cases.CENTRE, 90, 70)
    s.contours = [_abi.Contour(f, 0.2, (255, 0, 0))]
    ref = oracle.render(s)
    assert gpu.set_slab_cells(slices * 30 * 28) == 0
    try:
        assert np.array_equal(gpu.render(s), ref)
        assert np.array_equal(gpu.render(s), ref)
    finally:
        gpu.set_slab_cells(178956970)  # the default
