"""Fragments settled without FP64 and compared exactly where their depths are
near: scenes where many depths tie or nearly tie, objects beyond the table of
a frame, fields of different grids in one frame, cells far smaller and far
larger than a pixel.  The image is the oracle's, and the self-check (the
reference's arithmetic beside every single-precision decision) counts nothing."""
import numpy as np
import pytest

from contour3d_gb300 import _abi, fields
from . import cases

pytestmark = pytest.mark.gpu
COLORS = [(255, 0, 0), (0, 255, 0), (0, 0, 255), (255, 255, 0), (0, 255, 255), (255, 0, 255), (200, 200, 200),
          (90, 160, 30), (30, 90, 160)]


def _scene(levels, size=(150, 110), shape=(22, 18, 26), camera=cases.CAM0, view_height=1.0, grids=None, lines=False):
    f = fields.blobs(shape, nblobs=6, seed=3)
    s = _abi.make_scene(camera, cases.CENTRE, *size, view_height=view_height)
    s.contours = [_abi.Contour(f, lv, COLORS[q % 9], grids=grids) for q, lv in enumerate(levels)]
    if lines:
        s.lines = _abi.cube_edges(nitems=3, width=3.0)
    return s


def _stretched(n, a, b):
    u = np.arange(n, dtype=np.float64) / float(n - 1)
    return a + (b - a) * (u + 0.25 * u * (1.0 - u))


def _two_fields():
    s = _scene([0.5], lines=True)
    g, std = fields.modes((19, 23, 17), nmodes=8, kmin=1, kmax=3, power=1.0, seed=22)
    s.contours += [_abi.Contour(g, 0.1 * std, COLORS[1]), _abi.Contour(g, 0.1 * std, COLORS[2])]
    return s


def _plane():
    """Iso-planes through the camera axis: every triangle on it is seen edge on."""
    k, j, i = np.meshgrid(np.arange(9), np.arange(11), np.arange(13), indexing="ij")
    s = _abi.make_scene((0.5, 2.5, 0.5), cases.CENTRE, 61, 41)
    s.contours = [_abi.Contour(i - 6.0 + 0.0 * (j + k), 0.25, COLORS[0]),
                  _abi.Contour(k - 4.0 + 0.0 * (j + i), 0.0, COLORS[1])]
    return s


SCENES = {
    "same_surface_three_times": lambda: _scene([0.5, 0.5, 0.5], lines=True),
    "depths_within_1e-9": lambda: _scene([0.5, 0.5 + 1e-10, 0.5 - 1e-9, 0.5 + 1e-7, 0.5 - 1e-6]),
    "nine_objects": lambda: _scene([0.3 + 0.05 * q for q in range(9)], lines=True),
    "two_fields": _two_fields,
    "edge_on_planes": _plane,
    "one_pixel": lambda: _scene([0.4, 0.6], size=(1, 1)),
    "cells_below_a_pixel": lambda: _scene([0.5], size=(24, 18), shape=(60, 64, 56)),
    "cells_above_a_pixel": lambda: _scene([0.45, 0.55], size=(700, 500), shape=(7, 6, 8)),
    "far_camera": lambda: _scene([0.5], camera=(60.0, 45.0, 30.0), view_height=20.0),
    "stretched_grid": lambda: _scene([0.5, 0.6], grids=(_stretched(26, 0.0, 1.0), _stretched(18, 0.2, 0.7),
                                                        _stretched(22, 0.45, 0.55))),
    "descending_grid": lambda: _scene([0.5], grids=(_stretched(26, 1.0, 0.0), _stretched(18, 0.0, 1.0),
                                                    _stretched(22, 0.0, 1.0))),
}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_image_and_self_check(gpu, oracle, name):
    scene = SCENES[name]()
    ref = oracle.render(scene)
    assert np.array_equal(gpu.render(scene), ref)
    assert np.array_equal(gpu.render(scene), ref)  # unsynchronised
    img, _ = gpu.render(scene, with_depth=True)    # every depth exact
    assert np.array_equal(img, ref)
    gpu.set_filter_check(True)
    try:
        assert np.array_equal(gpu.render(scene), ref)
        st = gpu.stats()
    finally:
        gpu.set_filter_check(False)
    assert list(st.filter_violations) == [0] * 5 and st.shade_violations == 0


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_device_fields_of_two_grids(gpu, oracle, dtype):
    """Objects of different device fields in one frame, one surface drawn from both."""
    import torch
    a = fields.blobs((22, 18, 26), nblobs=6, seed=3)
    b, std = fields.modes((19, 23, 17), nmodes=8, kmin=1, kmax=3, power=1.0, seed=22)
    if dtype == "f32":
        a, b = a.astype(np.float32), b.astype(np.float32)
    dev = [torch.from_numpy(x).cuda() for x in (a, b, a.copy())]
    levels = [0.5, 0.2 * float(std), 0.5]
    scene = _abi.make_scene(cases.CAM0, cases.CENTRE, 150, 110)
    fl = []
    for t, lv, col in zip(dev, levels, COLORS):
        nz, ny, nx = t.shape
        fl.append((t.data_ptr(), 0 if dtype == "f64" else 1, (nx, ny, nz), [_abi.unit_grid(n) for n in (nx, ny, nz)],
                   lv, col))
    out = torch.empty(150 * 110 * 3, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    scene.contours = [_abi.Contour(x.astype(np.float64), lv, col) for x, lv, col in zip((a, b, a), levels, COLORS)]
    ref = oracle.render(scene)
    scene.contours = []
    for _ in range(2):
        assert gpu.render_device(scene, fl, out.data_ptr()) == 0
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().reshape(110, 150, 3), ref)
