"""Double-precision shading of every pixel of a field with a converter, its
triangles shared by the pixels of a warp and the list entries of a block: one
pixel, fewer than a warp, cells far larger and far smaller than a pixel, more
distinct triangles than a warp takes at a time.  The image is the oracle's."""
import numpy as np
import pytest

from contour3d_gb300 import _abi, fields
from . import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (5, 3), (33, 17), (97, 64), (300, 220)], ids=str)
@pytest.mark.parametrize("shape", [(5, 4, 6), (20, 26, 23)], ids=str)
def test_converter_image(gpu, oracle, size, shape):
    f, std = fields.modes(shape, nmodes=10, kmin=1, kmax=4, power=1.0, seed=11)
    s = _abi.make_scene(cases.CAM0, cases.CENTRE, *size)
    s.contours = [_abi.Contour(f, 0.2 * std, (250, 130, 7), converter="warp"),
                  _abi.Contour(f, -0.6 * std, (9, 90, 255), converter="warp")]
    ref = oracle.render(s)
    assert np.array_equal(gpu.render(s), ref)
    assert np.array_equal(gpu.render(s), ref)  # unsynchronised
