"""The gather on both sides of the line at 2^20 pixels (tiles counted whole) from which it runs with more
blocks per SM, against the oracle word for word."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N
from oracle.binding import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1016, 1023), (1024, 1024), (1025, 1023)])
def test_both_sides_of_the_line(cornell_c1_mesh, w, h):
    sc, mesh = cornell_c1_mesh
    cfg = g.default_config(w, height=h, photon_width=64, photon_height=48, hash_slots=4099,
                           radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.05)
    cam = g.look_at(sc.camera_origin, sc.camera_lookat, w, h, sc.fov)
    r = g.Renderer(cfg)
    r.upload_scene(mesh)
    r.set_camera(cam)
    o = Oracle(cfg, mesh.scene(), cam)
    r.run_passes(2)
    o.run_frames(2)
    for kind in ("flux_radius", "emission_n"):
        np.testing.assert_array_equal(np.ascontiguousarray(r.read_state(kind)).view(np.uint8),
                                      np.ascontiguousarray(o.read_state(kind)).view(np.uint8), err_msg=kind)
    r.close()
