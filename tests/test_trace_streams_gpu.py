"""Ray batches of one scene on several streams at once, and in a replayed graph
beside others, each larger than the lanes of the device (so that its rays are
dealt by a counter): the results are those of one batch after the other."""

import pytest

from snogray_b200 import Scene, scenes

pytestmark = pytest.mark.gpu

N = 1 << 21


class Batch:
    def __init__(self, seed):
        import torch
        self.rays = torch.from_numpy(scenes.random_rays(N, seed=seed)).cuda()
        self.prim = torch.empty(N, dtype=torch.int32, device="cuda")
        self.t = torch.empty(N, dtype=torch.float32, device="cuda")
        self.closest = N if seed % 2 else N // 2

    def clear(self):
        self.prim.fill_(-2)
        self.t.fill_(-1)

    def trace(self, sc, stream):
        sc.trace_device(self.rays.data_ptr(), N, self.closest, self.prim.data_ptr(), self.t.data_ptr(),
                        stream=stream.cuda_stream)

    def result(self):
        return self.prim.clone(), self.t.clone()


@pytest.fixture(scope="module")
def scene():
    with Scene(scenes.random_triangles(20_000, seed=1, edge_lo=0.01, edge_hi=0.1)) as sc:
        yield sc


def serial(sc, batches):
    import torch
    out = []
    for b in batches:
        b.clear()
        b.trace(sc, torch.cuda.current_stream())
        torch.cuda.synchronize()
        out.append(b.result())
    return out


def same(batches, want):
    import torch
    for b, (p, t) in zip(batches, want):
        assert torch.equal(b.prim, p) and torch.equal(b.t, t)


def test_batches_on_streams(scene):
    import torch
    batches = [Batch(s) for s in range(4)]
    want = serial(scene, batches)
    streams = [torch.cuda.Stream() for _ in batches]
    for _ in range(5):
        for b in batches:
            b.clear()
        torch.cuda.synchronize()
        for b, st in zip(batches, streams):
            b.trace(scene, st)
        torch.cuda.synchronize()
        same(batches, want)


def test_captured_batches_beside_others(scene):
    import torch
    batches = [Batch(s) for s in range(3)]
    want = serial(scene, batches)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        batches[0].trace(scene, main)
        batches[1].trace(scene, side)      # a branch of its own
        main.wait_stream(side)
    for _ in range(5):
        for b in batches:
            b.clear()
        torch.cuda.synchronize()
        graph.replay()
        batches[2].trace(scene, other)
        torch.cuda.synchronize()
        same(batches, want)
