"""The mixed path's kernels on both sides of the lines between their register bounds: 2^19 pixels for the eye
pass, 2^20 for the grid gather."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu


def render(sc, mesh, w, h, flags, passes):
    cfg = g.default_config(w, height=h, photon_width=128, photon_height=128, precision=N.PRECISION_MIXED, flags=flags,
                           radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.02)
    r = g.Renderer(cfg)
    r.upload_scene(mesh)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, w, h, sc.fov))
    r.run_passes(passes)
    r.synchronize()
    return r


@pytest.mark.parametrize("w,h", [(1016, 515), (1024, 512), (1024, 516)])
def test_the_eye_pass_on_both_sides(cornell_c1_mesh, w, h):
    """Its triangles are the plain path's (at most ten rays of half a million may differ: a closer
    near-coincident triangle that the plain walk's rounded box test skips)."""
    sc, mesh = cornell_c1_mesh
    a = render(sc, mesh, w, h, 0, 1)
    cfg = g.default_config(w, height=h, photon_width=128, photon_height=128, radius_rule=N.RADIUS_DIAGONAL,
                           radius_fraction=0.02)
    b = g.Renderer(cfg)
    b.upload_scene(mesh)
    b.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, w, h, sc.fov))
    b.run_passes(1)
    b.synchronize()
    assert (a.read_state("hit_triangle") != b.read_state("hit_triangle")).sum() <= 10
    a.close()
    b.close()


@pytest.mark.parametrize("w,h", [(1016, 1023), (1024, 1024), (1032, 1020)])
def test_the_grid_gather_on_both_sides(cornell_c1_mesh, w, h):
    """The gathered counts N are sums of alpha * M: double-float (48 bits) and IEEE double values of the same
    sums, relative difference below 2^-40."""
    sc, mesh = cornell_c1_mesh
    a = render(sc, mesh, w, h, N.FLAG_PHOTON_GRID, 2)
    b = render(sc, mesh, w, h, N.FLAG_PHOTON_GRID | N.FLAG_FP64_STATISTICS, 2)
    na, nb = (np.asarray(r.read_state("stats_n"), np.float64).reshape(-1) for r in (a, b))
    a.close()
    b.close()
    assert na.max() > 0
    assert (np.abs(na - nb) <= 2.0 ** -40 * np.abs(nb)).all()
