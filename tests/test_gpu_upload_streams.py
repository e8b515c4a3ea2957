"""Staged scene uploads on every kind of stream a renderer can be given: its own, a created one and the
per-thread handle, which names another stream in each staging thread. The frame rendered right after the
call is the one of the scene uploaded from the device."""
import numpy as np
import pytest

from _parity import PKG
from test_gpu_upload import frame, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["own", "created", "per-thread"])
def test_frame_after_upload(kind):
    import torch
    n, w, h = 400_003, 96, 64
    created = torch.cuda.Stream()
    r = PKG.GpsRenderer(w, h, 1)
    if kind != "own":
        r.set_stream(created.cuda_stream if kind == "created" else 2)  # 2: cudaStreamPerThread
    for seed in (1, 2, 3):  # each upload replaces another scene
        sp = scene(n, seed)
        sh = np.random.default_rng(seed).normal(0, 0.05, n * 9).astype(np.float32)
        r.set_gaussians_sh(sp, sh, 1)
        got, st = frame(r)
        g, s = torch.from_numpy(sp).cuda(), torch.from_numpy(sh).cuda()
        torch.cuda.synchronize()
        r.set_gaussians_device(g.data_ptr(), n, s.data_ptr(), sh.size, 1)
        want, stats = frame(r)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and st == stats
    r.close()
