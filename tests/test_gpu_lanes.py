"""Unsynchronised frames around the size at which a slab's objects stop taking
two lanes: just below it, just above it (pairs of objects after one another on
one stream, the next pair in the lists of the last), and a field whose slabs
change from one to two with the short last one.  Every frame, recorded ones
too, equals the synchronised one."""
import numpy as np
import pytest

from contour3d_gb300 import _abi, workloads
from . import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,levels,slabs", [((386, 390, 395), 3, 3), ((400, 402, 404), 3, 3),
                                                ((400, 402, 404), 5, 5), ((470, 640, 640), 3, 6)], ids=str)
def test_frames_equal_synchronised(gpu, shape, levels, slabs):
    import torch
    f, _ = workloads.modes_device(gpu, shape, nmodes=16, kmin=1, kmax=8, seed=5, dtype=torch.float32)
    lv = workloads.quantile_levels(f, np.random.default_rng(1), levels)
    nz, ny, nx = shape
    grids = [_abi.unit_grid(n) for n in (nx, ny, nz)]
    scene = _abi.make_scene(cases.CAM0, cases.CENTRE, 640, 360)
    out = torch.zeros(640 * 360 * 3, dtype=torch.uint8, device="cuda")
    pack = gpu.frame(scene, [(f.data_ptr(), 1, (nx, ny, nz), grids, t, workloads.PALETTE[q % len(workloads.PALETTE)])
                             for q, t in enumerate(lv)], out.data_ptr())
    torch.cuda.synchronize()

    def frame():
        out.zero_()
        torch.cuda.synchronize()
        assert gpu.render_pack(pack) == 0
        torch.cuda.synchronize()
        return out.cpu().numpy()

    gpu.set_async(False)
    try:
        ref = frame()
    finally:
        gpu.set_async(True)
    assert np.any(ref) and gpu.stats().slabs == slabs
    for _ in range(4):
        assert np.array_equal(frame(), ref)
        assert gpu.stats().unsynchronised == 1
    assert gpu.stats().graph == 2
