"""The bins the sorted path launches with (the runtime faked, fake_cudart.cpp): a tuned shape is the shape used,
whatever the frame; by default the renderer chooses; what is read back can be set again; a cached tuning
of the sorted path from before the sizes meant what they say is measured anew."""
import importlib
import json

from _fake_cuda import run
from conftest import load_package


def test_settings_select_what_they_name():
    run("""
fake.fake_watch.argtypes = [C.c_char_p, C.c_int, C.c_size_t]
fake.fake_watched.restype = C.POINTER(C.c_uint32 * 4)
fake.fake_watch(b"gpsb::k_sp_project", 1, 16)  # tw, th, tiles_x, tiles_y


def bins(w, h, r):
    r.render_sorted(PKG.OrbitCamera(distance=4.0).to_camera(w, h), P, 1)
    return tuple(fake.fake_watched().contents)[:2]


auto = PKG.gps.BLEND_TILE_AUTO
for w, h in ((64, 48), (1280, 720), (2600, 1700)):
    r = PKG.GpsRenderer(w, h, 1)
    r.set_gaussians(scene(100))
    before = r.tuning()
    assert (before["blend_tile_w"], before["blend_tile_h"]) == (auto, auto)
    chosen = bins(w, h, r)
    for shape in ((16, 16), (32, 8), (32, 32), (64, 64)):
        r.set_tuning(blend_tile_w=shape[0], blend_tile_h=shape[1])
        assert (r.tuning()["blend_tile_w"], r.tuning()["blend_tile_h"]) == shape
        assert bins(w, h, r) == shape, (w, h, shape)
        r.set_tuning(sort_digit_bits=8)  # other fields keep it
        assert bins(w, h, r) == shape
    for shape in ((8, 8), (16, 32), (64, 32), (1, 16), (32, 1), (128, 128)):
        assert raises(lambda: r.set_tuning(blend_tile_w=shape[0], blend_tile_h=shape[1])) is not None
    r.set_tuning(**before)
    assert bins(w, h, r) == chosen
    r.close()
""")


def test_large_frames_choose_by_their_entries():
    run("""
fake.fake_watch.argtypes = [C.c_char_p, C.c_int, C.c_size_t]
fake.fake_poke.argtypes = [C.c_char_p, C.c_int, C.c_void_p, C.c_size_t]
fake.fake_watched.restype = C.POINTER(C.c_uint32 * 2)
for w, h, choice in ((2600, 1700, True), (1280, 720, False)):
    r = PKG.GpsRenderer(w, h, 1)
    r.set_gaussians(scene(100))
    cam = PKG.OrbitCamera(distance=4.0).to_camera(w, h)
    # entries with 32 and with 64 pixels, the bins
    for fine, coarse, side in ((10, 5, 32), (11, 5, 64), (3, 3, 32), (0, 0, 32), (40_000, 10_001, 64)):
        both = (C.c_uint64 * 2)(fine, coarse if choice else 0)
        fake.fake_poke(b"gpsb::k_sp_project", 9, both, 16)
        for arg in (3, 4):
            fake.fake_watch(b"gpsb::k_blend<8, 8>", arg, 4)
            r.render_sorted(cam, P, 1)
            assert fake.fake_watched().contents[0] == (side if choice else 32), (w, fine, coarse, arg)
        fake.fake_watch(b"gpsb::k_entries", 5, 4)  # as many entries as that size has
        r.render_sorted(cam, P, 1)
        assert fine == 0 or fake.fake_watched().contents[0] == (coarse if choice and side == 64 else fine)
    if choice:  # too many small bins, not too many large ones
        fake.fake_poke(b"gpsb::k_sp_project", 9, (C.c_uint64 * 2)((1 << 30) + 1, (1 << 30) + 1), 16)
        assert "2^30" in str(raises(r.render_sorted, cam, P, 1))
    r.close()
""")


def test_old_cache_entries_are_measured_anew(tmp_path, monkeypatch):
    pkg = load_package()
    at = importlib.import_module(pkg.__name__ + ".autotune")
    assert len({json.dumps(s, sort_keys=True) for s in at.SORTED_SPACE}) == len(at.SORTED_SPACE)
    best = {"sort_digit_bits": 8, "blend_tile_w": 64, "blend_tile_h": 64}
    runs = []
    monkeypatch.setattr(at, "tune", lambda *a, **k: (runs.append(k["sorted_path"]) or (dict(best), [(best, 1.0)])))

    class R:
        def size(self):
            return 64, 48

        def set_tuning(self, **kw):
            self.set = kw

    path = tmp_path / "cache.json"
    p = pkg.RenderParams()
    old = {"best": {"sort_digit_bits": 8, "blend_tile_w": 32, "blend_tile_h": 32}, "ms": {}}
    particle = {"best": {"particle_items": 8, "particle_blocks_per_sm": 4}, "ms": {}}
    path.write_text(json.dumps({at.key(100, 64, 48, p.method, True): old, at.key(100, 64, 48, p.method, False): particle}))
    r = R()
    for _ in range(2):  # once: the new entry is used afterwards
        assert at.tuned(r, [], p, 100, sorted_path=True, cache_path=str(path)) == best and r.set == best
    assert at.tuned(r, [], p, 100, sorted_path=False, cache_path=str(path)) == particle["best"]
    assert runs == [True]
