"""Samples that are not finite: an image takes them by the filter's rule (a
weight of zero skips a sample; under a negative weight a component below -0.1
scales the sample so that the smallest is -0.1, which an infinite one turns into
NaN; the resolve clamps NaN to zero), restated in numpy."""

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes
from test_splat_gpu import mitchell1, synthetic_samples, write_all_done_checkpoint

pytestmark = pytest.mark.gpu


def restated(w, h, spp, result, jit):
    res = result.astype(np.float64).reshape(h + 4, w + 4, spp, 4)
    jt = jit.astype(np.float64).reshape(h + 4, w + 4, spp, 2)
    acc, wsum = np.zeros((h, w, 4)), np.zeros((h, w))
    ty, tx = np.mgrid[0:h, 0:w]
    with np.errstate(invalid="ignore", over="ignore"):
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                r, j = res[ty + dy + 2, tx + dx + 2], jt[ty + dy + 2, tx + dx + 2]
                wt = mitchell1(dx + j[..., 0] - 0.5) * mitchell1(dy + j[..., 1] - 0.5)
                tint = np.concatenate([r[..., :3] * r[..., 3:], r[..., 3:]], -1) * wt[..., None]
                least = np.fmin.reduce(tint[..., :3], -1)
                clamp = (wt < 0) & (least < -0.1)
                sc = np.where(clamp, -0.1 / np.where(clamp, least, 1.0), 1.0)
                used = wt != 0
                acc += np.where(used[..., None], tint * sc[..., None], 0.0).sum(2)
                wsum += np.where(used, wt * sc, 0.0).sum(2)
        scale = np.where((wsum > 0) & (wsum != 1), 1.0 / np.where(wsum > 0, wsum, 1.0), 1.0)
        acc *= scale[..., None]
        al = np.fmin(np.fmax(acc[..., 3], 0), 1)
        rgb = np.fmax(acc[..., :3], 0)
        return np.where(((al != 0) & (al != 1))[..., None], rgb / np.where(al > 0, al, 1.0)[..., None], rgb)


@pytest.mark.parametrize("spp", [1, 4])
@pytest.mark.parametrize("value", [(np.inf, 1, 1, 1), (np.inf, 0.5, np.inf, 1), (-np.inf, 1, 2, 1),
                                   (np.inf, -np.inf, 1, 1), (np.nan, 1, 1, 1), (np.nan, np.inf, 1, 0.5)])
def test_non_finite_samples(value, spp, tmp_path):
    w, h = 40, 20
    result, jit = synthetic_samples((w + 4) * (h + 4) * spp, seed=7)
    result[:, 3] = np.where(result[:, 3] == 0, 1, result[:, 3])
    at = (10 * (w + 4) + 20) * spp          # pattern pixel (20, 10): film pixel (18, 8)
    result[at], jit[at] = value, (0.3, 0.6)   # some weights below zero, none near it
    params = scenes.cornell_params(w, h, spp, seed=1)
    path = str(tmp_path / "a.ckp")
    with sb.Scene(scenes.cornell_box()) as sc:
        write_all_done_checkpoint(path, sc, scenes.cornell_camera(w, h), params, result, jit)
        with sb.Server(sb.engine_config(slots=1 << 16, item_paths=1 << 12)) as srv:
            img, st = srv.wait(srv.submit_resume(srv.add_scene(sc), path), timeout_ms=60000)
    assert st["status"] == sb.SNOG_OK
    want = restated(w, h, spp, result, jit)
    assert not np.isfinite(want).all() or (want[6:11, 16:21, 0] == 0).any()
    assert np.array_equal(np.isnan(img), np.isnan(want)) and np.array_equal(np.isinf(img), np.isinf(want))
    ok = np.isfinite(want)
    assert np.allclose(img[ok], want[ok], rtol=1e-3, atol=1e-4)
