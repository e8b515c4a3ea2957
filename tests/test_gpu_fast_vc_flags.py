"""ViewConditioned fast decisions with every set of flags, those compiled into a kernel of their own and the others:
frame and statistics equal the exact path's bit for bit."""
import numpy as np
import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radial,jitter,centre", [(r, j, c) for r in (False, True) for j in (False, True) for c in (False, True)])
def test_fast_equals_exact(radial, jitter, centre):
    from gps_pbvr_web_b200 import scenes
    splats, sh, deg = PKG.load_ply(scenes.cluster_scene(6000, seed=4, degree=1))
    cam = PKG.OrbitCamera(target=(0.0, 0.0, 0.0), distance=6.0, yaw=0.6, pitch=0.25, up=(0.0, -1.0, 0.0),
                          fov_y=0.9).to_camera(157, 91)
    p = PKG.RenderParams(spp_side=1, max_points_per_splat=512, method=PKG.Method.ViewConditioned)
    p.pbvr.radial_correction, p.pbvr.low_pass_jitter, p.pbvr.centre_depth, p.pbvr.base_k = radial, jitter, centre, 256.0
    out = []
    for mode in (0, 1):
        r = PKG.GpsRenderer(157, 91, 1)
        r.set_gaussians_sh(splats, sh, deg)
        r.set_fast_decisions(mode)
        r.render_ensembles(cam, p, 5, 3)
        st = r.read_stats()
        assert st.particles > 10_000
        out.append((r.read_accum(), (st.counters(), st.subpixel_writes)))
        r.close()
    assert np.array_equal(out[0][0].view(np.uint32), out[1][0].view(np.uint32)) and out[0][1] == out[1][1]
