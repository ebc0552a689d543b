"""Line segments whose few pixels per row or column are found from the line's
own equation, against the oracle: both major axes and the diagonal,
widths from 0 to wider than the image, ends far outside the screen."""
import numpy as np
import pytest

from contour3d_gb300 import _abi

pytestmark = pytest.mark.gpu


def _screen_lines(rng, n, spread, width):
    out = []
    for _ in range(n):
        p = rng.uniform(0.5 - spread, 0.5 + spread, (2, 3))
        out.append(_abi.Line(tuple(p[0]), tuple(p[1]), int(rng.integers(2, 6)), (255, 200, 40), width))
    return out


@pytest.mark.parametrize("size", [(1, 1), (97, 61), (61, 330)], ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("width", [0.0, 0.9, 2.0, 7.5, 1000.0])
def test_lines_match_oracle(gpu, oracle, size, width):
    rng = np.random.default_rng(int(10 * width) + size[0])
    # the camera looks along -y onto the plane's axes: exact horizontals and verticals
    s = _abi.make_scene((0.5, 3.0, 0.5), (0.5, 0.5, 0.5), *size)
    s.lines = [_abi.Line((0.1, 0.5, 0.4), (0.9, 0.5, 0.4), 3, (255, 0, 0), width),
               _abi.Line((0.3, 0.5, 0.1), (0.3, 0.5, 0.9), 2, (0, 255, 0), width),
               _abi.Line((0.1, 0.5, 0.1), (0.9, 0.5, 0.9), 2, (0, 0, 255), width)]
    s.lines += _screen_lines(rng, 12, 0.6, width) + _screen_lines(rng, 4, 30.0, width)
    assert np.array_equal(gpu.render(s), oracle.render(s))
