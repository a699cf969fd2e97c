"""The cells that an environment light's samples fall into, against a plain
bisection of the same cumulative distributions: light maps of two cells, of odd
sizes, downsampled, with black rows and columns, and one with negative texels,
whose distributions do not ascend.  The density of a sample names its cell; it
is three float products, so rtol 1e-6."""

import math

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes

F = np.float32


def distributions(env):
    """Row and column distributions as the scene builds them: sums in double,
    kept in float."""
    h, w = env.shape[:2]
    div = 1
    while w // div > 1024 or h // div > 1024:
        div += 1
    lw, lh = w // div, h // div
    lmap = np.zeros((lh, lw, 3), F)
    for y in range(h):
        ly = lh - y // div - 1
        for dx in range(div):
            if ly >= 0:
                part = env[y, dx:lw * div:div]
                lmap[ly, :len(part)] += part * F(1.0 / F(div * div))
    inten = (lmap[..., 0] + lmap[..., 1] + lmap[..., 2]) / F(3)
    lat, scale = -math.pi / 2 + math.pi / lh / 2, []
    for _ in range(lh):
        scale.append(math.cos(lat))
        lat += math.pi / lh
    bins = (inten.astype(np.float64) * np.array(scale)[:, None]).astype(F).astype(np.float64)
    row = np.cumsum(bins.reshape(-1) * (1 / np.cumsum(bins.reshape(-1))[-1]))[lw - 1::lw].astype(F)
    sums = np.cumsum(bins, 1)[:, -1:]
    col = np.cumsum(bins * np.where(sums == 0, 0, 1 / np.where(sums == 0, 1, sums)), 1).astype(F)
    return row, col


def bisect(a, v):
    lo, n = 0, len(a)
    while n:
        half = n // 2
        if a[lo + half] < v:
            lo, n = lo + half + 1, n - half - 1
        else:
            n = half
    return lo


def sky(w, h, kind):
    rng = np.random.default_rng(w * 1000 + h)
    env = rng.uniform(0.1, 1, (h, w, 3)).astype(F) ** 4
    if kind == "black":
        env[:h // 3] = 0
        env[:, w // 2:w // 2 + 2] = 0
    if kind == "negative":
        env[h // 2, w // 3] = -0.2 * env.sum() / (w * h)
        env[h // 4, w // 2] = -0.5
    return env


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,kind", [(2, 1, "plain"), (6, 3, "plain"), (34, 17, "black"), (64, 32, "black"),
                                      (66, 33, "negative"), (2050, 1025, "plain")])
def test_cells_equal_plain_bisection(w, h, kind):
    env = sky(w, h, kind)
    row, col = distributions(env)
    lh, lw = col.shape
    sd = scenes.SceneData(materials=scenes._mats([scenes.material(scenes.MAT_LAMBERT, (0.5, 0.5, 0.5))]),
                          vertices=[(-9, -9, 0), (9, -9, 0), (0, 9, 0)], triangles=[(0, 1, 2)], tri_mat=[0], envmap=env)
    rng = np.random.default_rng(7)
    n = 4000
    uv = rng.uniform(0, 1, (n, 2)).astype(F)
    edges_v = np.clip(rng.choice(row, n // 2), 0, 1)          # on a value, just below and just above
    uv[:n // 2, 1] = np.clip(np.nextafter(edges_v, rng.choice([-1, 1, 2], n // 2).astype(F)), 0, 1)
    uv[:n // 8, 1] = edges_v[:n // 8]
    rows = np.array([bisect(row, v) for v in uv[:, 1]])
    edges_u = np.clip(col[np.minimum(rows, lh - 1), rng.integers(0, lw, n)], 0, 1)
    uv[n // 4:3 * n // 4, 0] = edges_u[n // 4:3 * n // 4]
    uv[:2] = [(0, 0), (1, row[-1])]
    rows = np.array([bisect(row, v) for v in uv[:, 1]])
    probes = np.zeros((2 * n, 12), F)
    probes[:, 2] = np.repeat([1, -1], n)                       # from above, then from below
    probes[:, 6] = -probes[:, 2]
    probes[:, 7] = 10
    probes[:, 8:10] = 0.5
    probes[:, 10:12] = np.concatenate([uv, uv])
    with sb.Scene(sd) as sc:
        _, lights = sc.sample_probe(probes)
    seen = 0
    for k in range(n):
        r = rows[k]
        if r == lh:
            continue
        c = min(bisect(col[r], uv[k, 0]), lw - 1)
        y = r / lh + np.fmod(uv[k, 1], F(1) / F(lh))
        if abs(y - 0.5) < 1e-3 or not 1e-3 < y < 1 - 1e-3:
            continue
        got = lights[k if y > 0.5 else n + k, 0, 3]
        rp = row[r] - (row[r - 1] if r else F(0))
        cp = col[r, c] - (col[r, c - 1] if c else F(0))
        want = rp * cp * F(lw * lh) * F(0.25 / np.pi)
        np.testing.assert_allclose(got, want, rtol=1e-6, atol=1e-30, err_msg=f"{k} {uv[k]} row {r} col {c}")
        seen += 1
    assert seen > n // 4   # the half with a uniform v, less the strips left out
