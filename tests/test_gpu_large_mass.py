"""Holes so heavy that r^6 reaches the last powers of two (2^1022 to 2^1024), where the
straight-line reciprocal of the FP64 stages gives 0 without a mark (csrc/rt_fast_math.h):
one step of a scene scaled by 2^166 is the unit scene's step, scaled.  Powers of two
scale every operation but the roundings of a subnormal reciprocal (51 bits)."""
import numpy as np
import pytest

import relsim

pytestmark = pytest.mark.gpu
SCALE = 2.0 ** 166
R_OBS = 21.0  # r^6 = 2^1022.4 when scaled


def _camera(scale, precision):
    return relsim.make_camera(spin=0.5 * scale, mass=scale, r_obs=R_OBS * scale, incl_deg=70.0, fov_deg=30.0, width=16,
                              height=16, escape_radius=1000.0 * scale, disk_outer=20.0 * scale, max_steps=1, rtol=1e-3,
                              atol=1e-3, early_capture=False, precision=precision, critical_band=-1.0)


def _same_step(one, out):
    assert np.all(one["status"] == relsim.RAY_UNFINISHED) and np.all(one["steps_accepted"] == 1)
    for f in ("status", "steps_accepted", "steps_rejected"):
        np.testing.assert_array_equal(out[f], one[f])
    np.testing.assert_allclose(out["r"] / SCALE, one["r"], rtol=1e-13)
    for f in ("theta", "phi"):
        np.testing.assert_allclose(out[f], one[f], rtol=1e-13, atol=1e-13)
    # the step bends the rays: the ends' energies and angular momenta are those of the unit scene too
    np.testing.assert_allclose(out["dE"], one["dE"], rtol=0, atol=1e-13)
    np.testing.assert_allclose(out["dLz"] / SCALE, one["dLz"], rtol=0, atol=1e-12)


@pytest.mark.parametrize("precision", [relsim.PRECISION_FP64, relsim.PRECISION_MIXED])
def test_scaled_step(tracer, precision):
    # the unit scene in FP64: a scaled mixed camera is past the far zone's largest radius
    tracer.set_launch_config()
    one = tracer.dispatch(_camera(1.0, relsim.PRECISION_FP64), pixels=False)
    _same_step(one, tracer.dispatch(_camera(SCALE, precision), pixels=False))


def test_scaled_step_of_two_holes(tracer):
    tracer.set_launch_config()
    fields = ["status", "steps_accepted", "steps_rejected", "r", "theta", "phi", "dE", "dLz"]

    def scene(scale):
        body = relsim.make_source([6.0 * scale, 3.0 * scale, 0.0], mass=0.5 * scale, spin_parameter=0.3)
        return tracer.dispatch_multi(_camera(scale, relsim.PRECISION_FP64), [body], fields=fields, pixels=False)

    _same_step(scene(1.0), scene(SCALE))
