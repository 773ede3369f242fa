"""The persistent photon traversal of the 4-wide tree at the ends of its arithmetic, as
test_gpu_trace_wide has it for single rays: scenes from 2^-20 to 2^40 in size, far from the origin, and
rays with zero and tiny direction components.  The rays are the bounces of photons whose records are put
into a checkpoint (a mirror with no normal lets a photon go on as it came), and each hit is compared with
all triangles tested one by one."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N
from glslppm_gb300.renderer import MATERIAL_DTYPE
from tests.test_gpu_trace_wide import closest

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("precision", [N.PRECISION_MIXED, N.PRECISION_FP32])
@pytest.mark.parametrize("offset", [0.0, 37.0])
@pytest.mark.parametrize("power", [-20, 0, 20, 30, 40])
def test_no_entered_box_is_culled(power, offset, precision):
    rng = np.random.default_rng(power + 200)
    n, pw, ph, scale = 333, 80, 50, F(2.0) ** F(power)
    rays = pw * ph
    mid = rng.uniform(-1, 1, (n, 1, 3))
    pos = ((mid + rng.uniform(-0.3, 0.3, (n, 3, 3)) + offset).astype(F) * scale).astype(F)
    mats = np.zeros(1, MATERIAL_DTYPE)
    mats["color"], mats["brdf"] = 1.0, 1
    mesh = g.Mesh.from_arrays(pos, np.zeros(n, np.int32), mats).build_bvh()
    r = g.Renderer(g.default_config(8, photon_width=pw, photon_height=ph, precision=precision))
    r.upload_scene(mesh)
    at = float(F(offset) * scale)
    r.set_camera(g.look_at((at, at, at + 3 * float(scale)), (at, at, at), 8, 8, 45.0))
    r.set_tuning(wide_bvh=1, trace_blocks_per_sm=1)
    r.run_passes(1)
    r.synchronize()
    org = ((rng.uniform(-1.5, 1.5, (rays, 3)) + offset).astype(F) * scale).astype(F)
    d = rng.normal(size=(rays, 3))
    for axis in range(3):
        tiny = rng.choice([0.0, -0.0, 1e-38, -1e-30, 1e-27, -1e-26, 1e-20, 1e-8], rays)
        d[:, axis] = np.where(rng.random(rays) < 0.3, tiny, d[:, axis])
    d[np.abs(d).max(1) < 1e-3] = (1, 0, 0)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    flat = np.zeros((rays, 1), F)
    records = {"photon_position": np.hstack([org, flat]), "photon_flux": np.ones((rays, 4), F) * F([1, 1, 1, 0]),
               "photon_direction": np.hstack([d, flat]), "photon_hit": np.zeros((rays, 2), np.int32)}
    blob = bytes(r.save_checkpoint())
    for kind, new in records.items():
        old = np.ascontiguousarray(r.read_state(kind)).tobytes()
        where = blob.find(old)
        assert where >= 0 and len(old) == new.nbytes, kind
        blob = blob[:where] + np.ascontiguousarray(new).tobytes() + blob[where + new.nbytes:]
    r.load_checkpoint(blob)
    r.run_passes(1)
    r.synchronize()
    org, d, slot = r.debug_photon_rays()
    tri = np.ascontiguousarray(r.read_state("photon_hit")).reshape(-1, 2)[slot, 0]
    r.close()
    assert len(slot) == rays and (np.abs(d) < 1e-15).any(1).sum() > rays // 4
    stored = mesh.arrays().positions
    strict, _ = closest(stored, org, d, F(1e-3))
    loose, _ = closest(stored, org, d, F(-1e-3))
    sure = strict == loose
    assert sure.sum() > rays // 2 and (strict[sure] >= 0).sum() > rays // 8
    np.testing.assert_array_equal(tri[sure], strict[sure])
