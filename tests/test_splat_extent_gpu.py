"""Images whose width or height is in the millions (an engine's jobs are bounded
by their paths alone): samples of one colour give an image of that colour."""

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes
from test_splat_gpu import write_all_done_checkpoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(2_097_121, 1), (1, 1_048_561), (3, 1_300_000)])
def test_long_images(w, h, tmp_path):
    n = (w + 4) * (h + 4)
    result = np.tile(np.array([[0.25, 0.5, 0.75, 1]], np.float32), (n, 1))
    jit = np.full((n, 2), 0.5, np.float32)
    path = str(tmp_path / "a.ckp")
    with sb.Scene(scenes.cornell_box()) as sc:
        write_all_done_checkpoint(path, sc, scenes.cornell_camera(64, 64), scenes.cornell_params(w, h, 1, seed=1),
                                  result, jit)
        with sb.Server(sb.engine_config(slots=1 << 16, item_paths=1 << 16)) as srv:
            img, st = srv.wait(srv.submit_resume(srv.add_scene(sc), path), timeout_ms=60000)
    assert st["status"] == sb.SNOG_OK and img.shape == (h, w, 3)
    assert np.allclose(img, [0.25, 0.5, 0.75], rtol=1e-5)
