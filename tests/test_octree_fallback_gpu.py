"""Scenes whose tree the device builder does not take go to the host builder,
records included; scenes around the size from which the device builds, with
degenerate triangles and other primitives among them, are the same either way."""

import numpy as np
import pytest

import snogray_b200 as sb
import spec
from snogray_b200 import Scene, scenes

pytestmark = pytest.mark.gpu


def same(a, b, rays):
    ta, tb = a.octree(), b.octree()
    for k in ("children", "heads", "list", "origin"):
        assert np.array_equal(ta[k], tb[k]), k
    assert ta["size"] == tb["size"]
    pa, ha, na, ca = a.trace(rays, rays.shape[1] // 2, want_normal=True)
    pb, hb, nb, cb = b.trace(rays, rays.shape[1] // 2, want_normal=True)
    assert np.array_equal(pa, pb) and np.array_equal(ha, hb) and np.array_equal(na, nb) and ca == cb
    return pa


def test_root_grown_too_often_for_the_device():
    sd = scenes.random_triangles(5000, seed=3, edge_lo=0.01, edge_hi=0.05)
    v = sd.vertices.copy()
    v[0:3] = np.array([[0.5, 0.5, 0.5], [0.5 + 1e-6, 0.5, 0.5], [0.5, 0.5 + 1e-6, 0.5]], np.float32)
    v[-3:] = np.array([[1e7, 0, 0], [1e7, 1e6, 0], [1e7, 0, 1e6]], np.float32)
    sd.vertices = v
    rays = scenes.random_rays(4000, seed=4)
    with pytest.raises(sb.SnogError):
        Scene(sd, octree=Scene.OCTREE_DEVICE)
    with Scene(sd) as auto, Scene(sd, octree=Scene.OCTREE_HOST) as host:
        prim = same(auto, host, rays)
    assert np.array_equal(prim, spec.port_trace(sd, rays, rays.shape[1] // 2, threads=2)[0])
    assert (prim >= 0).any()


@pytest.mark.parametrize("n", [4000, 4095, 4096, 5000])
def test_sizes_around_the_device_builder(n):
    sd = scenes.mixed_scene(n - 200, 100, 100, seed=n)
    sd.vertices[3 * 17 + 1] = sd.vertices[3 * 17]        # degenerate triangles, the first among them
    sd.vertices[1] = sd.vertices[0]
    rays = scenes.random_rays(5000, seed=5)
    with Scene(sd) as auto, Scene(sd, octree=Scene.OCTREE_HOST) as host, \
            Scene(sd, octree=Scene.OCTREE_DEVICE) as dev:
        same(auto, host, rays)
        same(dev, host, rays)
