"""The eye pass that loads both next nodes before it tests its own (launches of up to 2^18 pixels) and the
one of larger images, against the oracle word for word: trees of one to nine triangles, where a step
ahead has no node to load, the reflecting and refracting materials, and images on both sides of the line."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N, scenes
from oracle.binding import Oracle

pytestmark = pytest.mark.gpu


def compare(sc, mesh, w, h, frames):
    cfg = g.default_config(w, height=h, photon_width=48, photon_height=32, hash_slots=997,
                           radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.02)
    cam = g.look_at(sc.camera_origin, sc.camera_lookat, w, h, sc.fov)
    r = g.Renderer(cfg)
    r.upload_scene(mesh)
    r.set_camera(cam)
    o = Oracle(cfg, mesh.scene(), cam)
    r.run_passes(frames)
    o.run_frames(frames)
    for kind in ("hit_position", "hit_triangle", "emission_n", "eye_rng", "photon_hit", "flux_radius"):
        np.testing.assert_array_equal(np.ascontiguousarray(r.read_state(kind)).view(np.uint8),
                                      np.ascontiguousarray(o.read_state(kind)).view(np.uint8), err_msg=f"{w}x{h} {kind}")
    r.close()


@pytest.mark.parametrize("triangles", [1, 2, 3, 5, 9])
def test_the_smallest_trees(cornell_c1_mesh, triangles):
    sc, mesh = cornell_c1_mesh
    a = mesh.arrays()
    light = int(a.light_triangles[0])
    others = [t for t in range(len(a.material_ids)) if a.materials["brdf"][a.material_ids[t]] != -1]
    ids = np.array([light] + others[:: max(1, len(others) // 8)][: triangles - 1])
    compare(sc, g.Mesh.from_arrays(a.positions[ids], a.material_ids[ids], a.materials).build_bvh(), 37, 29, 12)


@pytest.mark.parametrize("w,h", [(64, 48), (512, 512), (513, 512)])
def test_both_sides_of_the_line(w, h):
    sc = scenes.materials_box()
    compare(sc, sc.to_mesh(), w, h, 1)
