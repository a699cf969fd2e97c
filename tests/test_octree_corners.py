"""Surfaces on a regular grid whose steps round differently from the octree's
halves: their boxes start on a node's corner and stick out of the node by a
rounding error, and so go down to the corner's child until a node's size is zero.
The host builder ends there (in a process of its own, with a limit on its memory,
as one that does not end would use all there is)."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import resource
resource.setrlimit(resource.RLIMIT_AS, (8 << 30, 8 << 30))
import numpy as np
import snogray_b200 as sb
from snogray_b200 import scenes
n = 97
corner = (np.arange(n, dtype=np.float32) * np.float32(0.01))[:, None, None]
v = corner + np.eye(3, dtype=np.float32)[None] * np.float32(0.005)
sd = scenes.random_triangles(n, seed=1)
sd.vertices = np.ascontiguousarray(v.reshape(-1, 3), np.float32)
with sb.Scene(sd, device=False) as sc:
    info = sc.info()
    plist = sc.octree()["list"]
listed = set(int(p) for p in plist if p >= 0)
assert listed == set(range(n)), "every surface is listed"
assert info["max_depth"] > 84 and info["n_nodes"] < 400 * n, info
"""


def test_boxes_on_corners_end():
    out = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
