"""The direct integrator in long shading blocks: small jobs, which alone are shaded
in short blocks, give the same images beside jobs that keep more than 2^21 paths
to be traced (up to the order of the atomic additions, rtol 1e-4 as in the
engine's other image tests).  Both kinds of shading kernel append surviving,
listed and spawned rays, and a job is finished when each of its rays is counted.

The ring of spawned rays (a quarter of the slots) must not fill up: a vertex then
keeps one of its two rays, which one depends on its neighbours in the queue, and
images agree in the mean only."""

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes

pytestmark = pytest.mark.gpu

SIZES = [(40, 32, 8), (1, 1, 3), (33, 17, 5), (64, 48, 16)]


# The large job's integrator; with the path integrator the direct one's kernels run
# both kinds.
@pytest.mark.parametrize("large", ["direct", "path"])
def test_small_direct_jobs_beside_a_large_job(large):
    def job(sc, w, h, spp, seed, integrator="direct"):
        p = (scenes.direct_params(w, h, spp, seed=seed, light_samples=2) if integrator == "direct"
             else scenes.cornell_params(w, h, spp, seed=seed))
        return sc, scenes.cornell_camera(w, h), p

    # glass spheres: each vertex on them spawns a second ray
    with sb.Scene(scenes.cornell_box()) as sc, sb.Scene(scenes.nested_glass_scene()) as glass:
        small = [job(s, w, h, spp, seed) for s in (sc, glass) for seed, (w, h, spp) in enumerate(SIZES)]
        config = sb.engine_config(slots=1 << 22, item_paths=1 << 9)
        with sb.Engine(config) as eng:
            alone = [eng.render([j])[0][0] for j in small]
        with sb.Engine(config) as eng:
            # just above 2^21 paths; its items are dealt in turn with the small jobs'
            images, st = eng.render([job(sc, 360, 364, 16, 99, large)] + small)
    for got, want in zip(images[1:], alone):
        np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5)
    assert np.isfinite(images[0]).all() and images[0].mean() > 0.05
    assert st["paths"] == 360 * 364 * 16 + 2 * sum(w * h * s for w, h, s in SIZES)
