"""Engine jobs on both sides of the size from which shading runs in long
blocks, and with odd path counts: the image of the plain renderer, whose
shading kernels have the same arithmetic, up to the order of the atomic additions
of shadow contributions (rtol 1e-4, as the engine's other image tests)."""

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import Scene, scenes


@pytest.mark.gpu
# paths: (width + 4) (height + 4) spp against 2^21 -- below, just above, and a
# queue that is filled several times
@pytest.mark.parametrize("width,height,spp,slots", [(507, 505, 8, 1 << 22), (511, 517, 8, 1 << 22),
                                                    (301, 299, 37, 1 << 18)])
def test_engine_equals_plain_around_long_blocks(width, height, spp, slots):
    sd = scenes.terrain_scene(64, n_spheres=20, env_w=64, env_h=32)
    cam = scenes.terrain_camera(width, height)
    p = scenes.terrain_params(width, height, spp, seed=5)
    with Scene(sd) as sc:
        want, _ = sc.render(cam, p)
        with sb.Engine(sb.engine_config(max_lights=1, slots=slots)) as eng:
            for _ in range(2):
                (got,), st = eng.render([(sc, cam, p)])
                np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5)
    assert st["paths"] == width * height * spp


@pytest.mark.gpu
def test_jobs_of_several_sizes_in_long_blocks():
    """Blocks that hold paths of several jobs count each job's finished paths:
    every job completes, with the image of the plain renderer."""
    sd = scenes.terrain_scene(64, n_spheres=20, env_w=64, env_h=32)
    sizes = [(511, 517, 8), (1, 1, 3), (33, 17, 5), (301, 299, 9), (2, 63, 1), (7, 5, 64)]
    with Scene(sd) as sc:
        jobs = [(sc, scenes.terrain_camera(w, h), scenes.terrain_params(w, h, spp, seed=i))
                for i, (w, h, spp) in enumerate(sizes)]
        want = [s.render(cam, p)[0] for s, cam, p in jobs]
        with sb.Engine(sb.engine_config(max_lights=1, slots=1 << 20, item_paths=1 << 9)) as eng:
            got, st = eng.render(jobs)
    for g, w in zip(got, want):
        np.testing.assert_allclose(g, w, rtol=1e-4, atol=1e-5)
    assert st["paths"] == sum(w * h * spp for w, h, spp in sizes)
