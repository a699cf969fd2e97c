"""The splat at the edges of its tiles (32 x 16 target pixels, samples split
among blocks on small images), and with an infinite sample, against the float64
restatement of test_splat_gpu."""

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes
from test_splat_gpu import ref_splat, synthetic_samples, write_all_done_checkpoint

pytestmark = pytest.mark.gpu


def splat(w, h, spp, result, jit, path):
    params = scenes.cornell_params(w, h, spp, seed=spp)
    with sb.Scene(scenes.cornell_box()) as sc:
        write_all_done_checkpoint(path, sc, scenes.cornell_camera(w, h), params, result, jit)
        with sb.Server(sb.engine_config(slots=1 << 16, item_paths=1 << 12)) as srv:
            img, st = srv.wait(srv.submit_resume(srv.add_scene(sc), path), timeout_ms=60000)
    assert st["status"] == sb.SNOG_OK
    return img


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (1, 1, 9), (31, 15, 2), (32, 16, 3), (33, 17, 1), (64, 32, 5),
                                     (65, 33, 4), (3, 70, 6), (700, 3, 8), (160, 240, 4)])
def test_tile_edges(w, h, spp, tmp_path):
    result, jit = synthetic_samples((w + 4) * (h + 4) * spp, seed=w * 1000 + h + spp)
    img = splat(w, h, spp, result, jit, str(tmp_path / "a.ckp"))
    ref = ref_splat(w, h, spp, result, jit)
    assert np.allclose(img, ref, rtol=1e-3, atol=1e-4), np.abs(img - ref).max()


def test_infinite_sample_stays_within_the_filter(tmp_path):
    w, h, spp = 40, 20, 2
    result, jit = synthetic_samples((w + 4) * (h + 4) * spp, seed=3)
    at = (10 * (w + 4) + 20) * spp          # pattern pixel (20, 10): film pixel (18, 8)
    result[at] = (1, 1, 1, 1)
    ref = ref_splat(w, h, spp, result, jit)
    result[at] = (np.inf, 1, 1, 1)
    img = splat(w, h, spp, result, jit, str(tmp_path / "a.ckp"))
    far = np.ones((h, w), bool)
    far[6:11, 16:21] = False
    assert np.allclose(img[far], ref[far], rtol=1e-3, atol=1e-4)
    assert not np.isfinite(img[8, 18]).all()
