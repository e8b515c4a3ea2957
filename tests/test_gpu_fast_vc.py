"""ViewConditioned fast decisions from near to far: warps whose particles are all dropped by the keep draw, none of
them and some of them. Frame and statistics equal the exact path's bit for bit, and validation finds no
disagreement."""
import numpy as np
import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distance", [2.0, 12.0, 60.0, 400.0])
@pytest.mark.parametrize("radial,jitter,spp", [(True, True, 1), (False, False, 2)])
def test_fast_equals_exact(distance, radial, jitter, spp):
    from gps_pbvr_web_b200 import scenes
    splats, sh, deg = PKG.load_ply(scenes.cluster_scene(6000, seed=4, degree=1))
    cam = PKG.OrbitCamera(target=(0.0, 0.0, 0.0), distance=distance, yaw=0.6, pitch=0.25, up=(0.0, -1.0, 0.0),
                          fov_y=0.9).to_camera(160, 90)
    p = PKG.RenderParams(spp_side=spp, max_points_per_splat=512, method=PKG.Method.ViewConditioned)
    p.pbvr.radial_correction, p.pbvr.low_pass_jitter, p.pbvr.base_k = radial, jitter, 256.0
    out = []
    for mode in (0, 1, 2):
        r = PKG.GpsRenderer(160, 90, spp)
        r.set_gaussians_sh(splats, sh, deg)
        r.set_fast_decisions(mode)
        r.render_ensembles(cam, p, 5, 3)
        st = r.read_stats()
        assert st.particles > 10_000
        out.append((r.read_accum(), (st.counters(), st.subpixel_writes)))
        assert r.debug_fast_counts()[1] == 0
        r.close()
    for acc, st in out[1:]:
        assert np.array_equal(acc.view(np.uint32), out[0][0].view(np.uint32)) and st == out[0][1]
