"""Device blocks that outlive the scene or call they were made for: a scene
destroyed while its rays are still being traced, threads that share the pool,
and the bound on what is kept."""

import threading

import numpy as np
import pytest

from snogray_b200 import Scene, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 70_000])     # octree on the host, on the device
def test_scene_destroyed_under_its_own_trace(n):
    import torch
    rays = torch.from_numpy(scenes.random_rays(1 << 20, seed=1)).cuda()
    k = rays.shape[1]
    stream = torch.cuda.Stream()

    def trace(seed, then):
        prim = torch.full((k,), -2, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        sc = Scene(scenes.random_triangles(n, seed=seed, edge_lo=0.02, edge_hi=0.1))
        sc.trace_device(rays.data_ptr(), k, k, prim.data_ptr(), stream=stream.cuda_stream)
        then(sc)
        torch.cuda.synchronize()
        return prim

    want = [trace(s, lambda sc: (torch.cuda.synchronize(), sc.close())) for s in (1, 2)]

    def replace(sc):
        sc.close()
        Scene(scenes.random_triangles(n, seed=7, edge_lo=0.02, edge_hi=0.1)).close()   # takes the same blocks

    for s in (1, 2):
        assert torch.equal(trace(s, replace), want[s - 1])


def test_threads_share_the_pool():
    rays = scenes.random_rays(20_000, seed=2)
    data = [scenes.random_triangles(500 + 300 * i, seed=i, edge_lo=0.02, edge_hi=0.1) for i in range(4)]
    want = []
    for d in data:
        with Scene(d) as sc:
            want.append(sc.trace(rays, 10_000)[0])
    bad = []

    def work(i):
        for _ in range(8):
            with Scene(data[i]) as sc:
                if not np.array_equal(sc.trace(rays, 10_000)[0], want[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_what_is_kept_is_bounded():
    import torch
    Scene(scenes.random_triangles(1000, seed=1)).close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for n in (2_000, 150_000, 900_000, 20_000):
        with Scene(scenes.random_triangles(n, seed=1)) as sc:
            sc.trace(scenes.random_rays(3 * n, seed=1), n)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= (256 << 20) + (64 << 20)   # the bound, and 2 MiB pages
