"""The 4-wide walk's box test where a plane's scaled reciprocal is just short of overflowing: large scenes
and direction components that put 2^(e+15) / d of a node's exponent e within a per cent of the largest
float, on both sides of it.  Every ray is compared with all triangles tested one by one (test_gpu_trace_wide)."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N
from glslppm_gb300.renderer import MATERIAL_DTYPE
from tests.test_gpu_trace_wide import closest

pytestmark = pytest.mark.gpu
F = np.float32
FLT_MAX = float(np.finfo(F).max)


@pytest.mark.parametrize("power", [34, 36, 38, 40])
def test_no_entered_box_is_culled(power):
    rng = np.random.default_rng(power + 300)
    n, rays, scale = 333, 8000, F(2.0) ** F(power)
    mid = rng.uniform(-1, 1, (n, 1, 3))
    pos = ((mid + rng.uniform(-0.3, 0.3, (n, 3, 3))).astype(F) * scale).astype(F)
    mats = np.zeros(1, MATERIAL_DTYPE)
    mats["color"] = 0.5
    mesh = g.Mesh.from_arrays(pos, np.zeros(n, np.int32), mats).build_bvh()
    r = g.Renderer(g.default_config(8, photon_width=8, photon_height=8, precision=N.PRECISION_MIXED))
    r.upload_scene(mesh)
    org = (rng.uniform(-1.0, 1.0, (rays, 3)).astype(F) * scale).astype(F)
    d = rng.normal(size=(rays, 3))
    axis = rng.integers(0, 3, rays)
    d[np.arange(rays), axis] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    e = rng.integers(power - 9, power - 4, rays)  # the exponents of the scene's larger nodes
    share = rng.choice([0.45, 0.499, 0.502, 0.55, 0.99, 0.993, 0.995, 0.997, 0.999, 0.9999, 1.001, 1.01], rays)
    d[np.arange(rays), axis] = rng.choice([-1.0, 1.0], rays) * 2.0 ** (e + 15.0) / (share * FLT_MAX)
    d = d.astype(F)
    stored = mesh.arrays().positions
    strict, t = closest(stored, org, d, F(1e-3))
    loose, _ = closest(stored, org, d, F(-1e-3))
    sure = strict == loose
    tri, tg = r.debug_trace(org, d, photon=False, cull=False, mode=3)
    r.close()
    assert sure.sum() > rays // 2 and (strict[sure] >= 0).sum() > rays // 8
    lost = int((tri[sure] != strict[sure]).sum())
    assert lost == 0, (lost, int(sure.sum()))
    hit = sure & (strict >= 0)
    np.testing.assert_array_equal(tg[hit].view(np.uint32), t[hit].astype(F).view(np.uint32))
