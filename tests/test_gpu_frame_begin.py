"""The frame's start clears four hash slots a thread: jobs of a batch whose tables begin and end anywhere
within a thread's four, against the same jobs rendered alone, word for word."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu
KINDS = ("slot_winner", "slot_count", "photon_hit", "flux_radius", "eye_rng")


@pytest.mark.parametrize("sizes", [(1,), (3, 1, 1, 5), (4, 4096, 2), (997, 6, 7, 1, 1024, 3)])
@pytest.mark.parametrize("precision", [N.PRECISION_FP32, N.PRECISION_MIXED])
def test_tables_of_any_size(cornell_c1_mesh, sizes, precision):
    sc, mesh = cornell_c1_mesh
    cam = g.look_at(sc.camera_origin, sc.camera_lookat, 13, 11, sc.fov)
    cfgs = [g.default_config(13, height=11, photon_width=17, photon_height=9, hash_slots=n, seed=i + 1,
                             precision=precision, radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.05)
            for i, n in enumerate(sizes)]
    b = g.Batch(max_jobs=len(sizes), precision=precision)
    jobs = [b.add_job(c, mesh, cam) for c in cfgs]
    b.run_passes(12)
    b.synchronize()
    for c, j in zip(cfgs, jobs):
        r = g.Renderer(c)
        r.upload_scene(mesh)
        r.set_camera(cam)
        r.run_passes(12)
        r.synchronize()
        for k in KINDS:
            if k == "flux_radius" and precision == N.PRECISION_MIXED:
                continue
            np.testing.assert_array_equal(np.ascontiguousarray(b.read_state(j, k)).view(np.uint8),
                                          np.ascontiguousarray(r.read_state(k)).view(np.uint8), err_msg=k)
        r.close()
    b.close()
