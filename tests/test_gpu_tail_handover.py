"""trace_tail_lanes: walks are handed to the tail kernel once the ray queue is drained, not before.  With
few rays (spread over all warps) most warps still finish walks of their own first -- the walks that end in
the main kernel are the ones summed into the ray bins' costs -- and with many, walks are handed over in
their middle (node, closest hit and steps carried over): the same states, bit for bit."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu
KINDS = ("photon_position", "photon_flux", "photon_direction", "photon_hit", "photon_rng", "slot_winner", "slot_count",
         "flux_radius")


def renderer(sc, mesh, photons, **tuning):
    r = g.Renderer(g.default_config(32, photon_width=photons, photon_height=photons, radius_rule=N.RADIUS_DIAGONAL,
                                    radius_fraction=0.01))
    r.upload_scene(mesh)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, 32, 32, sc.fov))
    r.set_tuning(**tuning)
    return r


@pytest.mark.parametrize("lanes", [1, 8, 32])
@pytest.mark.parametrize("photons", [64, 128, 256])
def test_few_rays_are_not_handed_over_at_their_first_node(cornell_c1_mesh, photons, lanes):
    sc, mesh = cornell_c1_mesh
    r = renderer(sc, mesh, photons, trace_tail_lanes=lanes)
    r.run_passes(5)  # (before the first reorder, which clears the costs)
    segments = r.frame_info().photon_segments
    _, cost = r.debug_ray_bins()
    r.close()
    finished = int((cost & 0xFFFFFFFF).sum())
    # a warp hands over only after a lane of its own found the queue empty, so after at least one walk
    # has ended in it; a warp holds at most 32, and at these sizes fewer
    assert finished >= segments / 32, (finished, segments)


@pytest.mark.parametrize("tuning", [dict(trace_tail_lanes=1), dict(trace_tail_lanes=8),
                                    dict(trace_tail_lanes=32, trace_refill_steps=4),
                                    dict(trace_tail_lanes=32, unbinned_rays=1)])
def test_walks_handed_over_in_their_middle(cornell_c1_mesh, tuning):
    """One block per SM and 2^18 slots: every lane takes many rays before the queue is drained."""
    sc, mesh = cornell_c1_mesh
    states = []
    for t in (dict(), dict(trace_blocks_per_sm=1, **tuning)):
        r = renderer(sc, mesh, 512, **t)
        r.run_passes(3)
        r.synchronize()
        states.append({k: np.ascontiguousarray(r.read_state(k)).view(np.uint8) for k in KINDS})
        r.close()
    for k in KINDS:
        np.testing.assert_array_equal(states[0][k], states[1][k], err_msg=f"{tuning}: {k}")
