"""Inspection calls after a frame whose depths may be approximate: they draw
nothing, so however many there are they leave the frame's table of objects
alone.  In a process of its own, whose exit status counts too."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
from contour3d_gb300 import lib
from oracle.lib import Oracle
from tests import cases
gpu, oracle = lib.load(), Oracle()
scene = cases.blobs_small()
ref, want = oracle.render(scene), oracle.triangles(scene.contours[0])
assert np.array_equal(gpu.render(scene), ref)
for _ in range({calls}):
    got = gpu.triangles(scene.contours[0])
    assert got[1] == want[1] and got[0].tobytes() == want[0].tobytes()
assert np.array_equal(gpu.render(scene), ref)
print("complete")
"""


@pytest.mark.parametrize("calls", [1, 12])
def test_frames_and_inspection(gpu, oracle, calls):
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, calls=calls)], capture_output=True, text=True,
                       timeout=600)
    assert "complete" in r.stdout and r.returncode == 0, (r.returncode, r.stdout[-500:], r.stderr[-2000:])
