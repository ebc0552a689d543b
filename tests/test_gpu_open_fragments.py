"""More open fragments than the grid that settles them has lanes, so that whole
rounds of them are taken a lane each and the rest by fours: surfaces that
coincide, seen large, from one field and from two, and a converter's field in
one frame with others.  The image is the oracle's."""
import numpy as np
import pytest

from contour3d_gb300 import _abi, fields
from . import cases

pytestmark = pytest.mark.gpu
SIZE = (900, 700)
COLORS = [(255, 0, 0), (0, 255, 0), (0, 0, 255)]


@pytest.mark.parametrize("name", ["one_field", "two_fields", "converter"])
def test_long_lists(gpu, oracle, name):
    import torch
    f, std = fields.modes((20, 24, 22), nmodes=8, kmin=1, kmax=3, power=1.0, seed=22)
    b = fields.blobs((18, 21, 19), nblobs=6, seed=3)
    objs = {"one_field": [(f, 0.0, "identity")] * 3,
            "two_fields": [(f, 0.0, "identity"), (f.copy(), 0.0, "identity"), (f, 1e-9 * std, "identity")],
            "converter": [(b, 0.3, "identity"), (f, 0.0, "warp"), (f, -0.2 * std, "warp")]}[name]
    scene = _abi.make_scene((1.6, 1.4, 1.2), cases.CENTRE, *SIZE, view_height=0.6)
    scene.contours = [_abi.Contour(g, lv, col, converter=c) for (g, lv, c), col in zip(objs, COLORS)]
    ref = oracle.render(scene)
    scene.contours = []
    dev = {id(g): torch.from_numpy(g).cuda() for g, _, _ in objs}
    out = torch.zeros(ref.size, dtype=torch.uint8, device="cuda")
    fl = []
    for (g, lv, _), col in zip(objs, COLORS):
        nz, ny, nx = g.shape
        fl.append((dev[id(g)].data_ptr(), 0, (nx, ny, nz), [_abi.unit_grid(n) for n in (nx, ny, nz)], lv, col))
    pack = gpu.frame(scene, fl, out.data_ptr())
    for q, o in enumerate(objs):
        pack.fields[q].converter = gpu.converters[o[2]]
    torch.cuda.synchronize()
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        assert gpu.render_pack(pack) == 0
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)
    lanes = 32 * 16 * torch.cuda.get_device_properties(0).multi_processor_count
    assert gpu.stats().exact_fragments > 2 * lanes
