"""Device fields with converters in one frame: each has node positions of its
own, and a later field's must not stand in for an earlier one's where depths
are compared.  Two fields whose surfaces coincide up to 1e-9 (so that every
pixel of theirs is a near tie), with another field between them: the image is
the oracle's, pixel by pixel the nearer of the two."""
import numpy as np
import pytest

from contour3d_gb300 import _abi, fields
from . import cases

pytestmark = pytest.mark.gpu
SIZE = (150, 110)
RED, GREEN, BLUE = (255, 0, 0), (0, 255, 0), (0, 0, 255)


def _wavy(n, amp):
    g = _abi.unit_grid(n)
    return g + amp * np.sin(23.0 * g)


def _objects(between):
    """(field, grids, converter, level, colour) of every object, in drawing order."""
    a = fields.blobs((22, 18, 26), nblobs=6, seed=3)
    grids = tuple(_abi.unit_grid(n) for n in (26, 18, 22))
    near = tuple(_wavy(n, 1e-9) for n in (26, 18, 22))
    first = [(a, grids, "warp", 0.5, RED), (a, grids, "warp", 0.65, RED)]
    last = [(a.copy(), near, "warp", 0.5, GREEN)]
    if between == "larger":
        b, std = fields.modes((31, 35, 29), nmodes=8, kmin=1, kmax=3, power=1.0, seed=22)
        mid = [(b, None, "warp", 0.9 * std, BLUE)]
    elif between == "identity":
        b, std = fields.modes((19, 23, 17), nmodes=8, kmin=1, kmax=3, power=1.0, seed=22)
        mid = [(b, None, "identity", 0.9 * std, BLUE), (b, None, "identity", 0.9 * std * (1 + 1e-9), BLUE)]
    else:
        mid = []
    return first + mid + last


@pytest.mark.parametrize("between", ["nothing", "identity", "larger"])
@pytest.mark.parametrize("unsynchronised", [False, True])
def test_converters_keep_their_nodes(gpu, oracle, between, unsynchronised):
    import torch
    objs = _objects(between)
    scene = _abi.make_scene(cases.CAM0, cases.CENTRE, *SIZE)
    scene.lines = _abi.cube_edges(nitems=4, width=3.0) + [_abi.Line((0.2, 0.3, 0.4), (0.9, 0.6, 0.7), 5, width=4.0,
                                                                    converter="warp")]
    scene.contours = [_abi.Contour(f, lv, col, grids=g, converter=c) for f, g, c, lv, col in objs]
    ref = oracle.render(scene)
    hue = ref.reshape(-1, 3)
    # the two near surfaces are both in the picture
    assert min(((hue[:, c] > 0) & (hue.sum(1) == hue[:, c])).sum() for c in (0, 1)) > 100
    scene.contours = []
    dev = {}
    for f, *_ in objs:
        if id(f) not in dev:
            dev[id(f)] = torch.from_numpy(f).cuda()
    out = torch.zeros(SIZE[0] * SIZE[1] * 3, dtype=torch.uint8, device="cuda")
    fl = []
    for f, g, _, lv, col in objs:
        nz, ny, nx = f.shape
        fl.append((dev[id(f)].data_ptr(), 0, (nx, ny, nz), g or [_abi.unit_grid(n) for n in (nx, ny, nz)], lv, col))
    pack = gpu.frame(scene, fl, out.data_ptr())
    for q, o in enumerate(objs):
        pack.fields[q].converter = gpu.converters[o[2]]
    torch.cuda.synchronize()
    gpu.set_async(unsynchronised)
    try:
        for step in range(3):
            out.zero_()
            torch.cuda.synchronize()
            assert gpu.render_pack(pack) == 0
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy().reshape(SIZE[1], SIZE[0], 3), ref), f"frame {step}"
    finally:
        gpu.set_async(True)
