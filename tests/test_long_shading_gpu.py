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
