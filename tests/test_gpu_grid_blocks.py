"""The counting-sort grid's gather in blocks of any tunable size (its own are at most 128 threads), with
double-float and IEEE double statistics, at images that do not fill the tiles and at photon densities
from one photon to batches of many records a cell: the same states, word for word."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu


def state(sc, mesh, w, h, pw, block, flags):
    cfg = g.default_config(w, height=h, photon_width=pw, photon_height=pw, precision=N.PRECISION_MIXED,
                           flags=flags | N.FLAG_PHOTON_GRID, radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.03)
    r = g.Renderer(cfg)
    r.upload_scene(mesh)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, w, h, sc.fov))
    if block:
        r.set_tuning(gather_block=block)
    r.run_passes(11)
    r.synchronize()
    out = {k: np.ascontiguousarray(r.read_state(k)).view(np.uint8) for k in ("stats_n", "stats_r2", "stats_tau")}
    r.close()
    return out


@pytest.mark.parametrize("flags", [0, N.FLAG_FP64_STATISTICS])
@pytest.mark.parametrize("w,h,pw", [(1, 1, 33), (7, 3, 64), (67, 45, 1), (67, 45, 160)])
def test_blocks_give_the_same_statistics(cornell_c1_mesh, flags, w, h, pw):
    sc, mesh = cornell_c1_mesh
    want = state(sc, mesh, w, h, pw, 0, flags)
    for block in (32, 64, 96, 128, 160, 256):
        got = state(sc, mesh, w, h, pw, block, flags)
        for k in want:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"block {block}: {k}")
