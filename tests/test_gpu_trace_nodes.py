"""The photon traversal on the sizes and nodes where its shortcuts could differ from the general
walk (the single-kernel photon pass, one thread per segment): launches with fewer rays than lanes,
whose rays are spread over the warps, and node boxes whose planes come in the other order.  Every
operation is the same correctly rounded one, so the states are equal word for word."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu

KINDS = ("photon_position", "photon_flux", "photon_direction", "photon_hit", "photon_rng", "slot_winner",
         "slot_count", "hit_triangle", "flux_radius")


def state(sc, scene, pw, ph, flags=0, passes=3):
    cfg = g.default_config(24, photon_width=pw, photon_height=ph, radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.02)
    cfg.flags |= flags
    r = g.Renderer(cfg)
    r.upload_scene(scene)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, 24, 24, sc.fov))
    r.run_passes(passes)
    r.synchronize()
    out = {k: r.read_state(k) for k in KINDS}
    r.close()
    return out


def assert_same(a, b, what):
    for k in KINDS:
        np.testing.assert_array_equal(np.ascontiguousarray(a[k]).view(np.uint8),
                                      np.ascontiguousarray(b[k]).view(np.uint8), err_msg=f"{what}: {k}")


# one ray; fewer rays than warps; one to 32 rays a warp; about as many as lanes (152 SMs x 9 x 128), and more
@pytest.mark.parametrize("pw,ph", [(1, 1), (31, 1), (64, 64), (97, 89), (311, 373), (418, 419), (512, 512)])
def test_few_rays_spread_over_the_warps(cornell_c1_mesh, pw, ph):
    sc, mesh = cornell_c1_mesh
    assert_same(state(sc, mesh, pw, ph), state(sc, mesh, pw, ph, N.FLAG_FUSED_PHOTON), f"{pw}x{ph}")


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_boxes_with_their_planes_swapped(cornell_c1_mesh, axis):
    """The box test takes each axis' nearer plane by minimum, so a box given as (max, min) is the same
    box, for rays of every ordering."""
    sc, mesh = cornell_c1_mesh
    want = state(sc, mesh, 96, 64)
    a = mesh.arrays()
    swap = np.random.default_rng(axis).random(len(a.node_bounds)) < 0.3
    b = a.node_bounds.copy()
    b[swap, axis], b[swap, 3 + axis] = a.node_bounds[swap, 3 + axis], a.node_bounds[swap, axis]
    a.node_bounds = b
    assert_same(state(sc, a, 96, 64), want, f"axis {axis}")
