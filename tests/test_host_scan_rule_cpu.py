"""Which count scan a batch launches (the runtime faked, fake_cudart.cpp): one splat a thread below 240 tiles of
2048 splats, counted over the batch's ensembles, eight from there on."""
from _fake_cuda import run


def test_rule():
    run("""
for n, ensembles, per_thread in ((1, 1, 1), (10_000, 1, 1), (239 * 2048, 1, 1), (239 * 2048 + 1, 1, 8), (560_000, 1, 8),
                                 (119 * 2048, 2, 1), (120 * 2048, 2, 8), (3 * 2048, 64, 1), (4 * 2048, 64, 8)):
    r = PKG.GpsRenderer(64, 48, 1)
    r.set_gaussians(scene(n))
    fake.fake_clear()
    r.render_ensembles(CAM, P, 1, ensembles)
    assert ("gpsb::k_count_scan<%d>" % per_thread) in fake.fake_kernels().decode(), (n, ensembles, fake.fake_kernels())
    r.close()
""")
