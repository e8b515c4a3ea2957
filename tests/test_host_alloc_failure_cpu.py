"""Growing a buffer set that runs out of device memory half-way (the runtime faked, fake_cudart.cpp): the call
reports it, and the next, smaller call allocates what is missing before it launches anything. Every
allocation of the growing call fails in turn; afterwards no kernel may get a null pointer. A frame buffer
that could not be had is refused by every call that needs it."""
from _fake_cuda import run


def test_an_error_is_reported_once():
    run("""
r = PKG.GpsRenderer(64, 48, 1)
r.set_gaussians(scene(4000))
fake.fake_fail_malloc(1)
assert "out of memory" in str(raises(r.set_gaussians, scene(100_000)))
r.reset_accum()  # the old scene is still there
r.render_ensembles(CAM, P, 1, 2)
r.set_gaussians(scene(500))
r.close()
""")


def test_sorted_buffers():
    run("""
r = PKG.GpsRenderer(64, 48, 1)
r.set_gaussians(scene(4000))
r.render_sorted(CAM, P, 1)
for k in range(1, 40):
    r.set_gaussians(scene(4000 + 4000 * k))
    fake.fake_fail_malloc(k)
    e = raises(r.render_sorted, CAM, P, 1)
    fake.fake_fail_malloc(-1)
    if e is None:
        break
    assert "out of memory" in str(e)
    r.set_gaussians(scene(500))
    fake.fake_clear()
    r.render_sorted(CAM, P, 1)
    # without entries, as here, their lists are null and never read
    bad = [x for x in nulls().split(";") if x and x not in ("gpsb::k_bin_ranges#0", "gpsb::k_blend<8, 8>#7")]
    assert fake.fake_launches() > 5 and not bad, (k, bad)
assert k > 5
r.close()
""")


def test_batch_buffers():
    run("""
r = PKG.GpsRenderer(64, 48, 1)
r.set_gaussians(scene(4000))
r.render_ensembles(CAM, P, 1, 2)
size = 2
for k in range(1, 10):
    size += 3
    fake.fake_fail_malloc(k)
    e = raises(r.render_ensembles, CAM, P, 1, size)
    fake.fake_fail_malloc(-1)
    if e is None:
        break
    assert "out of memory" in str(e)
    fake.fake_clear()
    r.render_ensembles(CAM, P, 1, 1)
    assert fake.fake_launches() > 3 and not nulls(), (k, nulls())
assert k > 2
r.close()
""")


def test_denoiser_buffers():
    run("""
from gps_pbvr_web_b200 import denoise
net = denoise.NativeDenoiser()
r = PKG.GpsRenderer(64, 48, 1)
r.set_gaussians(scene(500))
net.render(r, CAM, P, 1, ensembles=2, gate_limit=10.0)
for k in range(1, 60):
    w, h = 64 + 8 * k, 48
    big = PKG.GpsRenderer(w, h, 1)
    big.set_gaussians(scene(500))
    big.render_ensembles(CAM, P, 1, 2)  # its own buffers are there
    fake.fake_fail_malloc(k)
    failed = False
    try:
        net.render(big, CAM, P, 1, ensembles=2, gate_limit=10.0)
    except Exception as e:
        assert "out of memory" in str(e), e
        failed = True
    fake.fake_fail_malloc(-1)
    big.close()
    if not failed:
        break
    fake.fake_clear()
    net.render(r, CAM, P, 1, ensembles=2, gate_limit=10.0)  # the frame size of before
    assert fake.fake_launches() > 20 and not nulls(), (k, nulls())
assert k > 10
""")


def test_frame_buffer():
    run("""
r = PKG.GpsRenderer(64, 48, 1)
r.set_gaussians(scene(500))
r.render_ensembles(CAM, P, 1, 2)
fake.fake_fail_malloc(1)
assert "out of memory" in str(raises(r.resize, 128, 96, 1))
fake.fake_clear()
cam = PKG.OrbitCamera(distance=4.0).to_camera(128, 96)
own = np.zeros((128 * 96, 4), np.float32)
OUT = own.ctypes.data
for call in (r.reset_accum, lambda: r.render_ensembles(cam, P, 1, 2), lambda: r.render_sorted(cam, P, 1),
             lambda: r.composite(P), r.read_accum):
    assert raises(call) is not None
r.render_trajectory([cam], P, 1, 2, OUT)  # into the caller's buffer
assert not nulls(), nulls()
r.resize(128, 96, 1)  # the same size again: there is room now
r.reset_accum()
r.render_ensembles(cam, P, 1, 2)
r.composite(P)
assert not nulls(), nulls()
r.close()
""")
