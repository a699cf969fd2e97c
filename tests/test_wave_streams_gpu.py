"""The plain renderer in several waves, on streams of the caller's and from several
threads at once, which share one pool of buffers and one stream for shadow rays:
the image of one wave whose kernels run one after the other, up to the order of
the atomic additions of shadow contributions (rtol 1e-4, atol 1e-5, as the
renderers' other tests)."""

import threading

import numpy as np
import pytest

import snogray_b200 as sb
from snogray_b200 import scenes

pytestmark = pytest.mark.gpu

JOBS = [(64, 48, 4, 1), (97, 61, 9, 2), (33, 90, 5, 3)]


def job(w, h, spp, seed):
    return scenes.cornell_camera(w, h), scenes.cornell_params(w, h, spp, seed=seed)


@pytest.fixture(scope="module")
def want():
    """With the kernels' times asked for, no launch runs beside another."""
    with pytest.MonkeyPatch.context() as m, sb.Scene(scenes.cornell_box()) as sc:
        m.setenv("SNOG_PROFILE_KERNELS", "1")
        return [sc.render(*job(*j))[0] for j in JOBS]


def render_on(sc, stream, k, out):
    import torch
    cam, p = job(*JOBS[k])
    img = torch.empty((p.height, p.width, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    sc.render_device(cam, p, img.data_ptr(), stream.cuda_stream)
    out.append((k, img))


# paths of a wave: a few rows' (the smallest wave there is), some rows', everything
@pytest.mark.parametrize("paths", [256, 2000, 20_000, 1 << 20])
def test_waves_on_a_stream(want, paths, monkeypatch):
    import torch
    monkeypatch.setenv("SNOG_WAVE_PATHS", str(paths))
    out = []
    with sb.Scene(scenes.cornell_box()) as sc:
        for k in range(len(JOBS)):
            render_on(sc, torch.cuda.Stream(), k, out)
        torch.cuda.synchronize()
    for k, img in out:
        np.testing.assert_allclose(img.cpu().numpy(), want[k], rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("shared", [True, False])
def test_threads_over_one_pool(want, shared):
    import torch
    n = 4
    scs = [sb.Scene(scenes.cornell_box()) for _ in range(1 if shared else n)]
    out, errors = [], []

    def work(t):
        try:
            stream = torch.cuda.Stream()
            for i in range(6):
                render_on(scs[t % len(scs)], stream, (t + i) % len(JOBS), out)
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for s in scs:
        s.close()
    assert not errors
    assert len(out) == 6 * n
    for k, img in out:
        np.testing.assert_allclose(img.cpu().numpy(), want[k], rtol=1e-4, atol=1e-5)
