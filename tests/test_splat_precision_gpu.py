"""Rounding of the splat's sums against 64 bits, and their order.

The filter's input is given (a checkpoint whose paths are all finished, as in
test_splat_gpu), with radiance of one sign and no clamped sample, so that a
pixel's error is that of the sums.  Sample positions are float32 on the film,
as the device and the reference take them.

Bound: with u = 2^-24 the unit roundoff, one rounding of a value with a spread
mantissa has an rms error of about 0.4 u.  A pixel ends in four of them (the two
sums, the reciprocal, the product): 0.8 u.  A sample's 25 additions to a partial
sum wander by sqrt(25 / 3) x 0.4 u x 1.5 (negative lobes), and its two products
by less, and these average over the samples: below 0.5 u from 16 samples on.
Together about u; the bound is 2 u rms.  A single float32 chain of 25 products
per sample takes 5 u at 16 samples and grows with their square root.
"""

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes
from test_splat_gpu import mitchell1, write_all_done_checkpoint

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def positive_samples(n, seed):
    rng = np.random.default_rng(seed)
    result = np.ones((n, 4), np.float32)
    result[:, :3] = rng.uniform(0.2, 1.2, (n, 3))
    return result, rng.random((n, 2), dtype=np.float32)


def exact_image(w, h, spp, result, jit):
    res = result.reshape(h + 4, w + 4, spp, 4)
    jt = jit.reshape(h + 4, w + 4, spp, 2)
    ty, tx = np.mgrid[0:h, 0:w]
    acc, wsum = np.zeros((h, w, 3)), np.zeros((h, w))
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            r, j = res[ty + dy + 2, tx + dx + 2], jt[ty + dy + 2, tx + dx + 2]
            sx = (tx + dx).astype(np.float32)[..., None] + j[..., 0]
            sy = (ty + dy).astype(np.float32)[..., None] + j[..., 1]
            assert sx.dtype == np.float32
            wt = (mitchell1(sx.astype(np.float64) - (tx[..., None] + 0.5))
                  * mitchell1(sy.astype(np.float64) - (ty[..., None] + 0.5)))
            assert (r[..., :3].max(-1) * wt).min() > -0.1       # nothing is clamped
            acc += (r[..., :3].astype(np.float64) * wt[..., None]).sum(2)
            wsum += wt.sum(2)
    return acc / wsum[..., None]


def images(w, h, spp, result, jit, path, times):
    params = scenes.cornell_params(w, h, spp, seed=1)
    out = []
    with sb.Scene(scenes.cornell_box()) as sc:
        write_all_done_checkpoint(path, sc, scenes.cornell_camera(w, h), params, result, jit)
        with sb.Server(sb.engine_config(slots=1 << 16, item_paths=1 << 12)) as srv:
            slot = srv.add_scene(sc)
            for _ in range(times):
                img, st = srv.wait(srv.submit_resume(slot, path), timeout_ms=60000)
                assert st["status"] == sb.SNOG_OK
                out.append(img)
    return out


# The tall ones have more tiles than the device takes blocks at a time.
@pytest.mark.parametrize("w,h,spp", [(1, 17_800, 16), (1, 17_800, 40), (64, 48, 16), (64, 48, 256), (23, 17, 1000)])
def test_sums_round_as_partial_sums_do(w, h, spp, tmp_path):
    result, jit = positive_samples((w + 4) * (h + 4) * spp, seed=h + spp)
    img = images(w, h, spp, result, jit, str(tmp_path / "a.ckp"), 1)[0]
    want = exact_image(w, h, spp, result, jit)
    rms = np.sqrt(np.mean(((img - want) / want) ** 2))
    print(f"rms error {rms / U:.2f} u")
    assert rms <= 2 * U, rms / U


@pytest.mark.parametrize("w,h,spp", [(64, 48, 2), (64, 48, 256), (33, 40, 13), (256, 200, 9)])
def test_sums_repeat(w, h, spp, tmp_path):
    result, jit = positive_samples((w + 4) * (h + 4) * spp, seed=spp)
    first, *rest = images(w, h, spp, result, jit, str(tmp_path / "a.ckp"), 6)
    for img in rest:
        assert np.array_equal(img, first)
