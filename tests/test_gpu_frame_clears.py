"""The clears inside the frame's kernels: every frame must start from empty subpixels, an empty scan scratch and,
after a reset, an empty accumulator. Frames whose subpixel count is odd, of one pixel, larger than the few tiles
of a small scene clear by themselves, split into several batches; each after a frame that left its data
behind. Image, counters and subpixel words must equal those of a fresh renderer that renders one ensemble a batch."""
import numpy as np
import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu


def scene(n, seed):
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 16), np.float32)
    s[:, 0:3] = rng.uniform(-1.5, 1.5, (n, 3))
    s[:, 3] = rng.uniform(0.2, 1.0, n)
    s[:, 4:7] = rng.normal(-3.0, 0.6, (n, 3))
    s[:, 8:12] = rng.normal(size=(n, 4))
    s[:, 12:15] = rng.uniform(0, 1, (n, 3))
    return s


def frame(r, cam, p, seed, ens):
    r.reset_accum()
    r.reset_stats()
    r.render_ensembles(cam, p, seed, ens)
    return r.read_accum(), r.read_stats()


@pytest.mark.parametrize("method", [PKG.Method.Gps, PKG.Method.Extinction])
@pytest.mark.parametrize("w,h,side,n", [(1, 1, 1, 3), (33, 31, 1, 300), (31, 33, 3, 5000), (1921, 1081, 1, 2), (640, 360, 2, 300_000)])
@pytest.mark.parametrize("ens,batch", [(1, 1), (3, 3), (5, 2)])
def test_every_frame_starts_empty(method, w, h, side, n, ens, batch):
    p = PKG.RenderParams(spp_side=side, method=method)
    near = PKG.OrbitCamera(distance=3.0).to_camera(w, h)
    cam = PKG.OrbitCamera(distance=7.0, yaw=0.3).to_camera(w, h)
    s = scene(n, n)
    fresh = PKG.GpsRenderer(w, h, side)
    fresh.set_gaussians(s)
    fresh.set_tuning(ensemble_batch=1)
    want, st = frame(fresh, cam, p, 9, ens)
    words = fresh.debug_subpixels(0)  # of the last ensemble
    r = PKG.GpsRenderer(w, h, side)
    r.set_gaussians(s)
    r.set_tuning(ensemble_batch=batch)
    frame(r, near, p, 5, ens + 1)  # leaves its subpixels, scan scratch and sums behind
    got, sg = frame(r, cam, p, 9, ens)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert sg.counters() == st.counters() and sg.particles == st.particles and sg.subpixel_writes == st.subpixel_writes
    assert np.array_equal(r.debug_subpixels((ens - 1) % batch), words)
    assert r.debug_error_word() == 0 and fresh.debug_error_word() == 0
    r.close()
    fresh.close()


def test_a_captured_frame_replays_like_a_launched_one():
    import torch

    w, h, n = 320, 200, 20_000
    p = PKG.RenderParams(spp_side=2)
    cam = PKG.OrbitCamera(distance=4.0).to_camera(w, h)
    r = PKG.GpsRenderer(w, h, 2)
    r.set_gaussians(scene(n, 3))
    stream = torch.cuda.Stream()
    r.set_stream(stream.cuda_stream)
    want, _ = frame(r, cam, p, 9, 3)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=stream):
        r.reset_accum()
        r.render_ensembles(cam, p, 9, 3)
    frame(r, cam, p, 2, 2)
    for _ in range(3):
        with torch.cuda.stream(stream):
            g.replay()
    assert np.array_equal(r.read_accum().view(np.uint32), want.view(np.uint32))
    assert r.debug_error_word() == 0
    del g
    r.close()
