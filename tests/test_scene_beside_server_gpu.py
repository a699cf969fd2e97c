"""Scenes that come and go while a server's worker thread captures its graphs
(on the first job of each kind) and renders: the jobs' images are those of a
server alone, and the scenes' rays hit what they hit alone."""

import threading

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes

pytestmark = pytest.mark.gpu


def serve(sc, jobs):
    with sb.Server(sb.engine_config(slots=1 << 18, item_paths=1 << 14)) as srv:
        slot = srv.add_scene(sc)
        ids = [srv.submit(slot, scenes.cornell_camera(p.width, p.height), p) for p in jobs]
        return [srv.wait(i, timeout_ms=60000)[0] for i in ids]


def test_scenes_destroyed_while_a_server_captures():
    jobs = [scenes.cornell_params(200, 160, 16, seed=1), scenes.direct_params(64, 64, 8, seed=2, light_samples=1),
            scenes.cornell_params(64, 48, 8, seed=3)]
    data = [scenes.random_triangles(n, seed=n, edge_lo=0.02, edge_hi=0.1) for n in (800, 6_000, 30_000)]
    rays = scenes.random_rays(20_000, seed=5)
    want_hits = []
    for d in data:
        with sb.Scene(d) as s:
            want_hits.append(s.trace(rays, 10_000)[0])
    stop, bad = threading.Event(), []

    def churn():
        while not stop.is_set():
            for d, w in zip(data, want_hits):
                with sb.Scene(d) as s:
                    if not np.array_equal(s.trace(rays, 10_000)[0], w):
                        bad.append(d)

    with sb.Scene(scenes.cornell_box()) as sc:
        want = serve(sc, jobs)
        t = threading.Thread(target=churn)
        t.start()
        try:
            for _ in range(6):
                for got, ref in zip(serve(sc, jobs), want):
                    # shadow rays add by float atomics, in any order
                    assert np.allclose(got, ref, rtol=1e-5, atol=1e-6)
        finally:
            stop.set()
            t.join()
    assert not bad
