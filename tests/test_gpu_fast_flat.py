"""Fast decisions of the GPS and ScreenOccupancy methods (gps_fast, so_fast in csrc/kernels.cu) and the
warp-unit particle loop: the validation mode finds no disagreement with the exact path, and the
fast mode's image, counters and subpixel words equal the exact mode's bit for bit. Sizes sit at the
edges of the loop: one particle, fewer than a warp's step, splats of one particle each, splats
of thousands; every subpixel side; sparse and dense ScreenOccupancy."""
import numpy as np
import pytest

from _parity import PKG, assert_bit_exact

pytestmark = pytest.mark.gpu
M = PKG.Method


def scene(n, seed, log_scale, opacity):
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 16), np.float32)
    s[:, 0:3] = rng.uniform(-1.5, 1.5, (n, 3))
    s[:, 3] = np.clip(opacity(rng, n), 0.0, 1.0)
    s[:, 4:7] = rng.normal(log_scale, 0.6, (n, 3))
    s[:, 8:12] = rng.normal(size=(n, 4))
    s[:, 12:15] = rng.uniform(0, 1, (n, 3))
    return s


SCENES = {
    "one": scene(1, 1, -3.0, lambda r, n: np.full(n, 0.7)),
    "few": scene(7, 2, -4.0, lambda r, n: r.uniform(0.1, 1.0, n)),
    "tiny splats": scene(20_000, 3, -6.0, lambda r, n: r.uniform(0.0, 0.3, n)),
    "mixed": scene(3_000, 4, -3.5, lambda r, n: 1.0 / (1.0 + np.exp(-r.normal(0.5, 2.0, n)))),
    "large opaque": scene(40, 5, -0.8, lambda r, n: np.where(r.random(n) < 0.5, 1.0, 0.999999)),
}


def render(r, cam, p, mode, ens):
    r.set_fast_decisions(mode)
    r.reset_accum()
    r.reset_stats()
    r.render_ensembles(cam, p, 21, ens)
    return r.read_accum(), r.read_stats(), r.debug_fast_counts(), r.debug_subpixels(0)


@pytest.mark.parametrize("name", list(SCENES))
@pytest.mark.parametrize("method,side,density", [(M.Gps, 1, 1.0), (M.Gps, 2, 1.0), (M.Gps, 3, 0.7), (M.Gps, 4, 2.0),
                                                  (M.ScreenOccupancy, 1, 1.0), (M.ScreenOccupancy, 2, 0.05),
                                                  (M.ScreenOccupancy, 3, 1.0), (M.ScreenOccupancy, 4, 3.0)])
def test_fast_equals_exact(name, method, side, density):
    w, h = (333, 187) if side < 3 else (129, 97)
    r = PKG.GpsRenderer(w, h, side)
    r.set_gaussians(SCENES[name])
    p = PKG.RenderParams(spp_side=side, method=method, density_scale=density)
    for d in (2.2, 6.0):
        cam = PKG.OrbitCamera(distance=d, yaw=0.4, pitch=0.2).to_camera(w, h)
        for ens in (1, 3):
            a0, s0, _, w0 = render(r, cam, p, 0, ens)
            a2, s2, (undecided, mismatch), w2 = render(r, cam, p, 2, ens)
            a1, s1, (ran, _), w1 = render(r, cam, p, 1, ens)
            assert mismatch == 0, (d, ens, mismatch, s0.particles)
            for a, s, sw in ((a1, s1, w1), (a2, s2, w2)):
                assert np.array_equal(a.view(np.uint32), a0.view(np.uint32)) and np.array_equal(sw, w0)
                assert s.counters() == s0.counters() and s.subpixel_writes == s0.subpixel_writes
                assert s.particles == s0.particles
            assert ran == undecided <= s0.particles
    assert r.debug_error_word() == 0
    r.close()


def test_most_particles_are_decided():
    r = PKG.GpsRenderer(1280, 720, 2)
    r.set_gaussians(SCENES["mixed"])
    cam = PKG.OrbitCamera(distance=4.0).to_camera(1280, 720)
    for method in (M.Gps, M.ScreenOccupancy):
        _, st, (undecided, mismatch), _ = render(r, cam, PKG.RenderParams(spp_side=2, method=method), 2, 2)
        assert mismatch == 0 and st.particles > 100_000 and undecided < 0.02 * st.particles, (method, undecided, st.particles)
    r.close()


@pytest.mark.parametrize("n,ens", [(1, 1), (255, 1), (256, 3), (257, 2), (2047, 1), (2049, 40), (75_000, 7), (75_000, 8)])
def test_count_scan_shapes(n, ens):
    """Both tile sizes of the count scan (one splat a thread below 296 tiles of 2048 splats, eight from there
    on): the counts of every splat and ensemble, the statistics and the image equal the CPU mirror's, with
    fixed counts, small and large means and capped splats among them."""
    s = scene(n, n, -6.0, lambda r, k: r.uniform(0.0, 1.0, k))
    s[: 1 + n // 5000, 4:7] = -2.0  # large means
    cam = PKG.OrbitCamera(distance=5.0).to_camera(160, 90)
    for method in (M.Gps, M.Extinction, M.ScreenOccupancy):
        assert_bit_exact(s, None, 0, 160, 90, 1, cam, PKG.RenderParams(spp_side=1, method=method, max_points_per_splat=500),
                         first_seed=5, count=ens)
