"""The launch counter (gpsb_profile.total_launches) against the kernels that were launched (the runtime faked,
fake_cudart.cpp), for the calls that count theirs."""
from _fake_cuda import run


def test_counts_are_the_kernels_launched():
    run("""
fake.fake_poke.argtypes = [C.c_char_p, C.c_int, C.c_void_p, C.c_size_t]
both = (C.c_uint64 * 2)(5000, 2000)  # bin entries of a sorted frame
fake.fake_poke(b"gpsb::k_sp_project", 9, both, 16)
L = PKG.abi.lib()
pairs = [np.zeros(700_000, np.uint32) for _ in range(4)]
ptr = [C.c_void_p(b.ctypes.data) for b in pairs]


def check(name, fn):
    before, l0 = r.profile()["total_launches"], fake.fake_launches()
    fn()
    got, want = r.profile()["total_launches"] - before, fake.fake_launches() - l0
    assert got == want and (want > 0 or name == "no pairs"), (name, got, want, fake.fake_kernels())
    fake.fake_clear()


for n, w, h in ((300, 64, 48), (2500, 2600, 1700)):
    r = PKG.GpsRenderer(w, h, 1)
    cam = PKG.OrbitCamera(distance=4.0).to_camera(w, h)
    r.set_gaussians(scene(n))
    out = np.zeros((2 * w * h, 4), np.float32)
    fake.fake_clear()
    check("reset", r.reset_accum)
    check("render", lambda: r.render_ensembles(cam, P, 1, 3))
    check("trajectory", lambda: r.render_trajectory([cam, cam], P, 1, 2, out.ctypes.data))
    for bits in (4, 6, 8):
        r.set_tuning(sort_digit_bits=bits)
        check("sorted", lambda: r.render_sorted(cam, P, 1))
        for pairs_n in (100, 700_000):
            check("sort", lambda: L.gpsb_sort_pairs(r.handle, *ptr, pairs_n, 24))
    check("no pairs", lambda: L.gpsb_sort_pairs(r.handle, *ptr, 0, 24))
    both[0] = both[1] = 0  # nothing visible: no entries to write and sort
    fake.fake_poke(b"gpsb::k_sp_project", 9, both, 16)
    check("sorted", lambda: r.render_sorted(cam, P, 1))
    both[0], both[1] = 5000, 2000
    fake.fake_poke(b"gpsb::k_sp_project", 9, both, 16)
    check("probe", lambda: r.probe_demand(cam, P))
    check("composite", lambda: r.composite(P))
    r.close()
""")
