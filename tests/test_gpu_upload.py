"""Scene uploads from pageable memory through the pinned staging threads (staged_upload in
csrc/renderer.cpp): the scene on the device is the caller's at the sizes where chunks begin and end, with and
without SH, from pinned memory too (which is copied directly), repeated on one renderer, and the
centroid (object zoom uses it) is the one of the direct path."""
import numpy as np
import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu
CHUNK = 512 << 10


def scene(n, seed):
    rng = np.random.default_rng(seed)
    s = rng.random((n, 16), dtype=np.float32) * 4 - 2
    s[:, 3] = rng.random(n)
    s[:, 4:7] = -4.0
    s[:, 8:12] += 0.1
    return s


def frame(r):
    p = PKG.RenderParams(spp_side=1, method=PKG.Method.Extinction)
    p.pbvr.calibration = PKG.Calibration.ObjectZoom
    r.reset_accum()
    r.reset_stats()
    r.render_ensembles(PKG.OrbitCamera(distance=6.0).to_camera(96, 64), p, 3, 2)
    return r.read_accum(), r.read_stats().counters()


@pytest.mark.parametrize("n", [16 * CHUNK // 64, 16 * CHUNK // 64 + 1, 17 * CHUNK // 64 - 1, 200_003])
@pytest.mark.parametrize("degree", [0, 1, 3])
def test_staged_equals_device_upload(n, degree):
    import torch
    per = (degree + 1) ** 2 - 1
    sp = scene(n, n)
    sh = np.random.default_rng(n + 1).normal(0, 0.05, n * 3 * per).astype(np.float32) if degree else None
    r = PKG.GpsRenderer(96, 64, 1)
    g = torch.from_numpy(sp).cuda()
    s = torch.from_numpy(sh).cuda() if degree else None
    torch.cuda.synchronize()
    r.set_gaussians_device(g.data_ptr(), n, s.data_ptr() if degree else None, sh.size if degree else 0, degree)
    want, stats = frame(r)
    pinned = torch.from_numpy(sp).pin_memory().numpy()
    for source in (sp, sp.copy(), pinned):
        if degree:
            r.set_gaussians_sh(source, sh, degree)
        else:
            r.set_gaussians(source)
        got, st = frame(r)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and st == stats
    r.set_gaussians(scene(10, 1))  # a small scene after a large one
    assert r.gaussian_count() == 10
    r.close()
