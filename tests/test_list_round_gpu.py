"""List rounds at their edges: node lists around one and two rounds' worth of
entries, hits of equal distance among them, batches around a warp's worth of
rays -- ids and distances equal to the oracle's restatement, bit for bit.

Every list entry is one of a few triangles repeated, so a ray's nearest
hit is shared by many entries of one list and the first in list order must be
the one kept; one other triangle in the middle of the list is in front of them
for part of the rays.
"""

import numpy as np
import pytest

import spec
from snogray_b200 import Scene, scenes


def stacked(n, front):
    """N triangles with one bounding box (so one list): all the same but number FRONT."""
    far = np.array([[0, 0, .25], [2, 0, .5], [0, 2, .5]], np.float32)
    near = np.array([[0, 2, .25], [2, 0, .25], [.3, .3, .5]], np.float32)
    v = np.concatenate([near if k == front else far for k in range(n)])
    return scenes.SceneData(materials=scenes.cornell_box().materials, vertices=v,
                            triangles=np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                            tri_mat=np.zeros(n, np.uint32))


def rays_through(n_rays, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((7, n_rays), np.float32)
    r[0], r[1], r[2] = rng.uniform(0, 1, n_rays), rng.uniform(0, 1, n_rays), -1
    r[3:5] = rng.uniform(-.02, .02, (2, n_rays))
    r[5], r[6] = 1, np.inf
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 131])
@pytest.mark.parametrize("n_rays", [1, 33, 700])
def test_long_lists_with_ties(n, n_rays):
    sd = stacked(n, n // 2)
    rays = rays_through(n_rays, n)
    for nc in (n_rays, n_rays // 2, 0):
        ref_prim, ref_t, _, ref, _ = spec.port_trace(sd, rays, nc, threads=1)
        with Scene(sd) as sc:
            prim, t, _, cnt = sc.trace(rays, nc)
        assert np.array_equal(prim, ref_prim)
        hit = np.nonzero(prim[:nc] >= 0)[0]
        assert np.array_equal(t[hit].view(np.uint32), ref_t[hit].view(np.uint32))
        assert cnt["closest_tests"] == ref["closest"]["surface_tests"]   # one node: every entry once


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [-1, 0])
def test_batches_around_a_full_device(fill):
    """Long lists along rays, one ray fewer than the device's trace lanes (8
    blocks of 128 per SM) and as many: entries dealt singly and in pairs."""
    import torch
    n = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 128 + fill
    sd = scenes.random_triangles(5000, seed=4, edge_lo=0.02, edge_hi=0.1)
    rays = scenes.random_rays(n, seed=6)
    nc = n // 2
    ref_prim, ref_t, _, _, _ = spec.port_trace(sd, rays, nc, threads=8)
    with Scene(sd) as sc:
        assert sc.info()["pair_lists"] == 1
        prim, t, _, _ = sc.trace(rays, nc)
        dev = torch.empty(n, dtype=torch.int32, device="cuda")
        sc.trace_device(torch.from_numpy(rays).cuda().data_ptr(), n, nc, dev.data_ptr())
        torch.cuda.synchronize()
    assert np.array_equal(prim, ref_prim) and np.array_equal(dev.cpu().numpy(), ref_prim)
    hit = np.nonzero(prim[:nc] >= 0)[0]
    assert np.array_equal(t[hit].view(np.uint32), ref_t[hit].view(np.uint32))
