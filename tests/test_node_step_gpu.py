"""Node visits where comparisons tie: lattice rays in all 26 directions of
{-1, 0, 1}^3 from the corners, edges and faces of octree cells, through a
scene whose cells have those corners -- midplanes met at equal distances, rays
in a midplane, zero direction components, every octant -- against the oracle's
restatement, ids and distances bit for bit.
"""

import itertools

import numpy as np
import pytest

import spec
from snogray_b200 import Scene, scenes


def lattice_scene(slant):
    """Triangles at the cells' centres of a 1/8 lattice over [0, 2]^3, the first spanning the whole cube;
    SLANT tilts them out of the axis planes."""
    v = [[[0, 0, 0], [2, 2, 0], [0, 2, 2]]]
    for c in itertools.product(range(0, 16, 3), repeat=3):
        p = np.array(c) / 8 + 1 / 16
        s = np.array([1, -1, 1]) * slant
        v.append([p - 1 / 32, p + [1 / 32, 1 / 32, -1 / 32] + s, p + [-1 / 32, 1 / 32, 1 / 32] - s])
    v = np.array(v, np.float32).reshape(-1, 3)
    n = len(v) // 3
    return scenes.SceneData(materials=scenes.cornell_box().materials, vertices=v,
                            triangles=np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                            tri_mat=np.zeros(n, np.uint32))


def lattice_rays(step, t_max):
    d = np.array([x for x in itertools.product((-1, 0, 1), repeat=3) if any(x)], np.float32)
    o = np.array(list(itertools.product(np.arange(-step, 2 + 2 * step, step), repeat=3)), np.float32)
    r = np.empty((7, len(o) * len(d)), np.float32)
    r[0:3] = np.repeat(o, len(d), 0).T
    r[3:6] = np.tile(d, (len(o), 1)).T
    r[6] = t_max
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("slant", [0.0, 1 / 64])
@pytest.mark.parametrize("step,t_max", [(0.25, np.inf), (0.1875, 1.0)])
def test_lattice_rays_match_restatement(slant, step, t_max):
    sd, rays = lattice_scene(slant), lattice_rays(step, t_max)
    n = rays.shape[1]
    for nc in (n, 0):
        ref_prim, ref_t, _, ref, _ = spec.port_trace(sd, rays, nc, threads=2)
        with Scene(sd) as sc:
            prim, t, _, cnt = sc.trace(rays, nc)
        assert np.array_equal(prim, ref_prim)
        hit = np.nonzero(prim[:nc] >= 0)[0]
        assert np.array_equal(t[hit].view(np.uint32), ref_t[hit].view(np.uint32))
        assert cnt["closest_nodes"] <= ref["closest"]["node_calls"]
        assert cnt["any_nodes"] <= ref["any"]["node_calls"]
        if nc:
            assert len(hit) > n // 50
