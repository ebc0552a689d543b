"""Approximate depths near the camera: cells that are not small against their
distance, seen from among them, so that a fragment may be several times nearer
than its cell's corner 0 (or farther).  The image is the oracle's, and in the
self-check every approximate depth lies within its bound, every bound within
the tolerance that near depths are told apart by."""
import numpy as np
import pytest

from contour3d_gb300 import _abi

pytestmark = pytest.mark.gpu
VIEWS = [(-1.0, -1.0, -1.0), (1.0, 1.0, 1.0), (-1.0, 0.2, 0.1), (0.3, -0.2, -1.0)]


def _scene(view, distance, nodes, seed):
    """A random field of `nodes` a side on the unit cube from its middle, 90 degrees from top to bottom."""
    view = np.asarray(view) / np.linalg.norm(view)
    camera = np.array([0.52, 0.47, 0.55]) - 0.3 * view
    right = np.cross(view, (0.0, 0.0, 1.0))
    right /= np.linalg.norm(right)
    w, h, size = 160, 120, 2.0 * distance
    s = _abi.Scene(tuple(camera), (0.5, 0.5, 0.5), (0.3, 2.0, -1.0), w, h, tuple(camera + distance * view),
                   tuple(right * size * w / h), tuple(np.cross(right, view) * size))
    f = np.random.default_rng(seed).random((nodes, nodes, nodes))
    s.contours = [_abi.Contour(f, 0.35, (255, 90, 20)), _abi.Contour(f, 0.7, (20, 90, 255))]
    return s


@pytest.mark.parametrize("view", VIEWS, ids=str)
@pytest.mark.parametrize("nodes", [5, 6, 9])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_bounds_near_the_camera(gpu, oracle, view, nodes, dtype):
    import torch
    scene = _scene(view, 0.02, nodes, 7)
    if dtype == "f32":
        for c in scene.contours:
            c.field = c.field.astype(np.float32).astype(np.float64)
    ref = oracle.render(scene)
    dev = torch.from_numpy(scene.contours[0].field).cuda()
    if dtype == "f32":
        dev = dev.float()
    grids = [_abi.unit_grid(nodes)] * 3
    fl = [(dev.data_ptr(), 0 if dtype == "f64" else 1, (nodes,) * 3, grids, c.threshold, c.color)
          for c in scene.contours]
    scene.contours = []
    out = torch.zeros(ref.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for check in (False, True):
        gpu.set_filter_check(check)
        try:
            assert gpu.render_device(scene, fl, out.data_ptr()) == 0
            st = gpu.stats()
        finally:
            gpu.set_filter_check(False)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)
    assert st.exact_fragments > 0
    assert list(st.filter_violations) == [0] * 5 and st.shade_violations == 0
