"""The 4-wide quantised walk's box test at the ends of its arithmetic: scenes from 2^-20 to 2^40 in
size (where the scaled reciprocals overflow), far from the origin, and rays with zero and tiny
direction components.  A culled box that the ray enters loses its closest hit, so every ray is compared
with all triangles tested one by one, in the same correctly rounded single-precision operations: the
same triangle at the same t, bit for bit.  Left out are the rays whose closest hit depends on rounding
at an edge (a barycentric within 1e-3 of 0, a few thousand times the operations' error)."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N
from glslppm_gb300.renderer import MATERIAL_DTYPE

pytestmark = pytest.mark.gpu
F = np.float32


def dot(a, b):
    return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]


def cross(a, b):
    x, y, z = a[..., 0], a[..., 1], a[..., 2]
    u, v, w = b[..., 0], b[..., 1], b[..., 2]
    return np.stack([y * w - v * z, z * u - w * x, x * v - u * y], -1)


def closest(pos, org, d, margin):
    v0, e0, e1 = pos[:, 0], pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0]
    with np.errstate(all="ignore"):
        o, d = org[:, None], np.broadcast_to(d[:, None], (len(d), len(pos), 3))
        pv = cross(d, np.broadcast_to(e1, d.shape))
        det = dot(np.broadcast_to(e0, d.shape), pv)
        tv = o - v0
        qv = cross(tv, np.broadcast_to(e0, d.shape))
        u, v, t = dot(tv, pv) / det, dot(d, qv) / det, dot(np.broadcast_to(e1, d.shape), qv) / det
        w = (F(1) - u) - v
    assert t.dtype == F
    ok = (u >= margin) & (v >= margin) & (w >= margin) & (t >= 0) & (t < F(1e20))
    t = np.where(ok, t, np.inf)
    k = t.argmin(1)
    tk = t[np.arange(len(t)), k]
    return np.where(np.isfinite(tk), k, -1), tk


@pytest.mark.parametrize("offset", [0.0, 37.0])
@pytest.mark.parametrize("power", [-20, 0, 20, 30, 40])
def test_no_entered_box_is_culled(power, offset):
    rng = np.random.default_rng(power + 100)
    n, rays, scale = 333, 4000, F(2.0) ** F(power)
    mid = rng.uniform(-1, 1, (n, 1, 3))
    pos = ((mid + rng.uniform(-0.3, 0.3, (n, 3, 3)) + offset).astype(F) * scale).astype(F)
    mats = np.zeros(1, MATERIAL_DTYPE)
    mats["color"] = 0.5
    mesh = g.Mesh.from_arrays(pos, np.zeros(n, np.int32), mats).build_bvh()
    r = g.Renderer(g.default_config(8, photon_width=8, photon_height=8, precision=N.PRECISION_MIXED))
    r.upload_scene(mesh)
    org = ((rng.uniform(-1.5, 1.5, (rays, 3)) + offset).astype(F) * scale).astype(F)
    d = rng.normal(size=(rays, 3))
    for axis in range(3):
        tiny = rng.choice([0.0, -0.0, 1e-38, -1e-30, 1e-27, -1e-26, 1e-20, 1e-8], rays)
        d[:, axis] = np.where(rng.random(rays) < 0.3, tiny, d[:, axis])
    d[np.abs(d).max(1) < 1e-3] = (1, 0, 0)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    stored = mesh.arrays().positions
    strict, t = closest(stored, org, d, F(1e-3))
    loose, _ = closest(stored, org, d, F(-1e-3))
    sure = strict == loose
    tri, tg = r.debug_trace(org, d, photon=False, cull=False, mode=3)
    r.close()
    assert sure.sum() > rays // 2 and (strict[sure] >= 0).sum() > rays // 8
    np.testing.assert_array_equal(tri[sure], strict[sure])
    hit = sure & (strict >= 0)
    np.testing.assert_array_equal(tg[hit].view(np.uint32), t[hit].astype(F).view(np.uint32))
