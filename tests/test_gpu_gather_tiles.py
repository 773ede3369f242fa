"""The gather's 8x4-pixel tiles at images that do not fill them, and its in-cell bounds from the table
and from the division (a radius so small that the grid has more cells than the table), against the
oracle word for word."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N
from oracle.binding import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (8, 4), (9, 5), (33, 31), (403, 3), (3, 129)])
@pytest.mark.parametrize("fraction", [0.05, 2e-5])
def test_tiles_against_the_oracle(cornell_c1_mesh, w, h, fraction):
    sc, mesh = cornell_c1_mesh
    cfg = g.default_config(w, height=h, photon_width=96, photon_height=64, hash_slots=997,
                           radius_rule=N.RADIUS_DIAGONAL, radius_fraction=fraction)
    cam = g.look_at(sc.camera_origin, sc.camera_lookat, w, h, sc.fov)
    r = g.Renderer(cfg)
    r.upload_scene(mesh)
    r.set_camera(cam)
    o = Oracle(cfg, mesh.scene(), cam)
    r.run_passes(12)
    o.run_frames(12)
    for kind in ("flux_radius", "emission_n", "hit_triangle", "slot_count"):
        np.testing.assert_array_equal(np.ascontiguousarray(r.read_state(kind)).view(np.uint8),
                                      np.ascontiguousarray(o.read_state(kind)).view(np.uint8), err_msg=kind)
    np.testing.assert_array_equal(r.read_image().view(np.uint32), o.read_image(0).astype(np.float32).view(np.uint32).reshape(h, w, 3))
