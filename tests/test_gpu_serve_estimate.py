"""What a served request holds before its triangles are known (code arrays,
cell words, the least triangle maps, the canvas) against the estimate that
admits it: a field without crossings holds nothing else, and buffers are
allocated a quarter larger than asked for."""
import numpy as np
import pytest

from contour3d_gb300 import _abi
from . import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unsynchronised", [0, 1])
@pytest.mark.parametrize("levels", [1, 2, 3])
def test_estimate_covers_what_is_held_without_triangles(gpu, levels, unsynchronised):
    import torch
    n = (150, 140, 160)
    field = torch.zeros(n[::-1], dtype=torch.float32, device="cuda")
    out = torch.zeros(64 * 48 * 3, dtype=torch.uint8, device="cuda")
    grids = [_abi.unit_grid(q) for q in n]
    scene = _abi.make_scene(cases.CAM0, cases.CENTRE, 64, 48)
    pack = gpu.frame(scene, [(field.data_ptr(), 1, n, grids, 1.0 + q, (255, 0, 0)) for q in range(levels)], out.data_ptr())
    torch.cuda.synchronize()
    assert gpu.lib.contour3d_gb300_set_server_async(unsynchronised) == 0
    try:
        with gpu.server(slots=1) as sv:
            for _ in range(2):
                st = sv.wait(sv.submit(pack))
    finally:
        gpu.lib.contour3d_gb300_set_server_async(0)
    torch.cuda.synchronize()
    assert not np.any(out.cpu().numpy())
    # unsynchronised frames also size the lists of candidates and tiny triangles (at least 2^20 and 2^16 entries)
    lists = unsynchronised * min(levels, 2) * ((1 << 20) * (16 + 8 + 2) + (1 << 18) + (1 << 20) * 48 // 8)
    assert 0 < st.held_bytes <= 1.25 * (st.estimate_bytes + lists) + (2 << 20), (st.held_bytes, st.estimate_bytes)
