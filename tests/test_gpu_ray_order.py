"""The order of the photon rays that the library chooses until shapes are set: sppm_get_tuning reports the
order and refill interval that ran, and setting what it reports changes neither."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N

pytestmark = pytest.mark.gpu
FP32, MIXED = N.PRECISION_FP32, N.PRECISION_MIXED


def renderer(sc, mesh, precision, pw=64, ph=48, flags=0):
    cfg = g.default_config(32, photon_width=pw, photon_height=ph, radius_rule=N.RADIUS_DIAGONAL, radius_fraction=0.01,
                           precision=precision)
    cfg.flags |= flags
    r = g.Renderer(cfg)
    r.upload_scene(mesh)
    r.set_camera(g.look_at(sc.camera_origin, sc.camera_lookat, 32, 32, sc.fov))
    return r


def binned(r):
    """Did the rays of the next passes go through the bins?"""
    r.run_passes(3)
    r.synchronize()
    _, cost = r.debug_ray_bins()
    return bool(cost.sum())


# the plain path bins a single job's rays from 3/4 * 2^20 slots on
@pytest.mark.parametrize("precision,pw,ph,order,refill", [(FP32, 64, 48, 1, 32), (FP32, 1024, 767, 1, 32),
                                                          (FP32, 1024, 768, 0, 32), (MIXED, 64, 48, 1, 4),
                                                          (MIXED, 1024, 768, 1, 4)])
def test_reports_what_ran_and_takes_it_back(cornell_c1_mesh, precision, pw, ph, order, refill):
    sc, mesh = cornell_c1_mesh
    r = renderer(sc, mesh, precision, pw, ph)
    assert binned(r) == (order == 0)
    t = r.get_tuning()
    assert (t.unbinned_rays, t.trace_refill_steps) == (order, refill)
    r.set_tuning(t)
    assert r.get_tuning().as_dict() == t.as_dict()
    assert binned(r) == (order == 0)
    r.set_tuning(**{**t.as_dict(), "gather_block": 64})  # one field of the report changed
    assert r.get_tuning().unbinned_rays == order and r.get_tuning().trace_refill_steps == refill
    assert binned(r) == (order == 0)
    r.close()


@pytest.mark.parametrize("precision", [FP32, MIXED])
def test_the_report_of_a_context_that_has_not_run(cornell_c1_mesh, precision):
    sc, mesh = cornell_c1_mesh
    r = renderer(sc, mesh, precision)
    r.set_tuning(r.get_tuning())
    assert not binned(r)
    r.close()


def test_an_order_that_is_set(cornell_c1_mesh):
    sc, mesh = cornell_c1_mesh
    for precision, tuning, want in ((FP32, dict(), (0, 32)), (MIXED, dict(), (0, 8)), (MIXED, dict(unbinned_rays=1), (1, 4)),
                                    (FP32, dict(unbinned_rays=1), (1, 32)), (FP32, dict(wide_bvh=1), (0, 8))):
        r = renderer(sc, mesh, precision)
        r.run_passes(1)
        r.set_tuning(**tuning)
        t = r.get_tuning()
        assert (t.unbinned_rays, t.trace_refill_steps) == want, (precision, tuning)
        assert binned(r) == (want[0] == 0)
        r.close()


def test_without_bins(cornell_c1_mesh):
    sc, mesh = cornell_c1_mesh
    r = renderer(sc, mesh, MIXED, flags=N.FLAG_UNBINNED_RAYS)
    r.run_passes(1)
    assert (r.get_tuning().unbinned_rays, r.get_tuning().trace_refill_steps) == (1, 4)
    r.set_tuning()
    assert (r.get_tuning().unbinned_rays, r.get_tuning().trace_refill_steps) == (1, 4)
    r.close()
