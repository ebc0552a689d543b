"""Vertices that are corners of their cells, and what the reference draws of
their triangles.  Edges whose values differ by less than 1e-8 keep the tail
corner, which depends on the triangle.  Levels equal to node values make
triangles without area, and the reference tests those at the border pixels
too when they lie off the image (both ends of its box are clamped).  The image
and the depths are the oracle's, and the self-check counts nothing."""
import numpy as np
import pytest

from contour3d_gb300 import _abi
from . import cases

pytestmark = pytest.mark.gpu


def _check(gpu, oracle, scene):
    ref, depth = oracle.render(scene, with_depth=True)
    assert np.array_equal(gpu.render(scene), ref)
    assert np.array_equal(gpu.render(scene), ref)  # unsynchronised
    img, d = gpu.render(scene, with_depth=True)
    assert np.array_equal(img, ref) and np.array_equal(d, depth, equal_nan=True)
    gpu.set_filter_check(True)
    try:
        assert np.array_equal(gpu.render(scene), ref)
        st = gpu.stats()
    finally:
        gpu.set_filter_check(False)
    assert list(st.filter_violations) == [0] * 5 and st.shade_violations == 0


@pytest.mark.parametrize("converter", ["identity", "warp"])
@pytest.mark.parametrize("scale", [1e-12, 3e-9, 2e-8])
def test_kept_tails(gpu, oracle, converter, scale):
    f = scale * np.random.default_rng(5).standard_normal((11, 9, 13))
    scene = _abi.make_scene(cases.CAM0, cases.CENTRE, 130, 90)
    scene.contours = [_abi.Contour(f, 0.1 * scale, (255, 120, 9), converter=converter),
                      _abi.Contour(f, -0.8 * scale, (9, 120, 255), converter=converter)]
    _check(gpu, oracle, scene)


@pytest.mark.parametrize("camera", [cases.CAM0, (-1.9, 1.7, 2.1), (0.5, 3.0, 0.6)], ids=str)
@pytest.mark.parametrize("view_height", [0.1, 0.3])
def test_triangles_without_area_off_the_image(gpu, oracle, camera, view_height):
    """A field of whole numbers seen through a window much smaller than it."""
    f = np.random.default_rng(8).integers(0, 4, size=(14, 12, 13)).astype(np.float64)
    scene = _abi.make_scene(camera, cases.CENTRE, 96, 64, view_height=view_height)
    scene.contours = [_abi.Contour(f, 1.0, (255, 255, 0)), _abi.Contour(f, 2.0, (0, 255, 0))]
    _check(gpu, oracle, scene)
