"""Colours settled in single precision: lights along, across and against the
surfaces' normals (clamped, free and at the limit of both), a direction of
length zero, colours whose channels truncate differently, and so few pixels
that a block of the double-precision pass holds a handful.  The image is the
oracle's, and no single-precision colour differs from the double one."""
import numpy as np
import pytest

from contour3d_gb300 import _abi, fields
from . import cases

pytestmark = pytest.mark.gpu
LIGHTS = [(0.0, 2.0, -1.0), (1.0, 0.0, 0.0), (-3.0, -2.0, 5.0), (1e-6, 1.0, 1e-6), (0.0, 0.0, 0.0)]


@pytest.mark.parametrize("light", LIGHTS, ids=str)
@pytest.mark.parametrize("size", [(9, 7), (130, 90), (420, 300)], ids=str)
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_colours(gpu, oracle, light, size, dtype):
    f = fields.blobs((22, 18, 26), nblobs=6, seed=5).astype(dtype).astype(np.float64)
    s = _abi.make_scene(cases.CAM0, cases.CENTRE, *size, light=light)
    s.contours = [_abi.Contour(f, 0.5, (255, 1, 128)),
                  _abi.Contour(f, 0.4, (7, 254, 200))]
    ref = oracle.render(s)
    assert np.array_equal(gpu.render(s), ref)
    gpu.set_filter_check(True)
    try:
        assert np.array_equal(gpu.render(s), ref)
        st = gpu.stats()
    finally:
        gpu.set_filter_check(False)
    assert st.shade_violations == 0
