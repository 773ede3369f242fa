"""The generator's step as the kernels form it (floors by a sum rounded down, fused operations where a
product is exact) against its separate operations in numpy, from states at the ends of their range,
fractional ones, and around the multiples of each lane's quotient, where the floors step."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu
F = np.float32
Q = np.array([1225, 1585, 2457, 2098], F)
R = np.array([1112, 367, 92, 265], F)
A = np.array([3423, 2646, 1707, 1999], F)
M = np.array([4194287, 4194277, 4194191, 4194167], F)
QINV = np.array([8.163265302e-04, 6.309148157e-04, 4.070004215e-04, 4.766444326e-04], F)


def step(s):
    beta = np.floor(s * QINV)
    p = A * (s - beta * Q) - beta * R
    return p + (np.sign(-p) * (F(0.5) * M) + F(0.5) * M)


def test_the_draws_of_an_emission(cornell_c1_mesh):
    sc, mesh = cornell_c1_mesh
    pw, ph = 256, 128
    rng = np.random.default_rng(5)
    s = rng.integers(0, 1 << 22, (ph * pw, 4)).astype(F)
    k = np.arange(ph * pw) % 3424
    edge = np.minimum(k[:, None] * Q + rng.integers(-1, 2, s.shape), F(1 << 22))
    s[: len(s) // 4] = np.maximum(edge, 0)[: len(s) // 4].astype(F)
    frac = slice(len(s) // 4, len(s) // 2)
    s[frac] = (rng.random((len(s) // 4, 4), F) * F(1 << 22) * rng.choice([1, 1e-3, 1e-6], (len(s) // 4, 4))).astype(F)
    s[-4:] = np.array([[0] * 4, [1] * 4, [1 << 22] * 4, [0.5] * 4], F)
    s[-8:-4] = M - np.arange(4)[:, None].astype(F)
    r = g.Renderer(g.default_config(8, photon_width=pw, photon_height=ph, radius_rule=N.RADIUS_DIAGONAL,
                                    radius_fraction=0.02))
    r.upload_scene(mesh)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, 8, 8, sc.fov))
    blob = bytes(r.save_checkpoint())
    seeds = np.ascontiguousarray(r.read_state("photon_rng")).tobytes()
    at = blob.find(seeds)
    assert at >= 0 and len(seeds) == s.nbytes
    r.load_checkpoint(blob[:at] + s.tobytes() + blob[at + s.nbytes:])
    r.run_passes(1)  # every slot emits: three draws on the light, two for the lobe
    r.synchronize()
    got = np.ascontiguousarray(r.read_state("photon_rng")).reshape(-1, 4)
    r.close()
    for _ in range(5):
        s = step(s)
    assert s.dtype == F
    np.testing.assert_array_equal(got.view(np.uint32), s.view(np.uint32))
