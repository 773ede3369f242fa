"""The walk that loads both next nodes before it tests its own (launches of up to 2^17 slots), at the
trees where a step ahead has no node to load -- one to nine triangles, the last node, the last
ordering -- and on both sides of the line, against the single-kernel photon pass: the same states, word
for word."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu
KINDS = ("photon_position", "photon_flux", "photon_direction", "photon_hit", "photon_rng", "slot_winner", "slot_count",
         "flux_radius")


def state(sc, scene, pw, ph, flags, passes=3):
    cfg = g.default_config(16, photon_width=pw, photon_height=ph, radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.02)
    cfg.flags |= flags
    r = g.Renderer(cfg)
    r.upload_scene(scene)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, 16, 16, sc.fov))
    r.run_passes(passes)
    r.synchronize()
    out = {k: np.ascontiguousarray(r.read_state(k)).view(np.uint8) for k in KINDS}
    r.close()
    return out


def compare(sc, scene, pw, ph):
    a, b = state(sc, scene, pw, ph, 0), state(sc, scene, pw, ph, N.FLAG_FUSED_PHOTON)
    for k in KINDS:
        np.testing.assert_array_equal(a[k], b[k], err_msg=f"{pw}x{ph}: {k}")


@pytest.mark.parametrize("triangles", [1, 2, 3, 5, 9])
def test_the_smallest_trees(cornell_c1_mesh, triangles):
    sc, mesh = cornell_c1_mesh
    a = mesh.arrays()
    light = int(a.light_triangles[0])
    others = [t for t in range(len(a.material_ids)) if a.materials["brdf"][a.material_ids[t]] != -1]
    ids = np.array([light] + others[:: max(1, len(others) // 8)][: triangles - 1])
    small = g.Mesh.from_arrays(a.positions[ids], a.material_ids[ids], a.materials).build_bvh()
    compare(sc, small, 61, 37)


@pytest.mark.parametrize("pw,ph", [(512, 256), (257, 511), (362, 363)])
def test_both_sides_of_the_line(cornell_c1_mesh, pw, ph):
    sc, mesh = cornell_c1_mesh
    compare(sc, mesh, pw, ph)
