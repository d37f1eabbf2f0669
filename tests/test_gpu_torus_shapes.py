"""Torus-shaded frames on both sides of the lines at which the trace's launch shape
changes (640 rays an SM, 2,048 for a hole of spin 0.98 and more): every ray's bytes are
those of its rows traced by themselves, in the shape of a small frame."""
import numpy as np
import pytest

import relsim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spin,per_sm", [(0.9, 639), (0.9, 641), (0.979, 700), (0.98, 700), (-0.98, 700), (0.998, 2049)])
def test_shapes_trace_the_same(tracer, spin, per_sm):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    width = 256
    rows = -(-per_sm * sms // width)
    kw = dict(spin=spin, r_obs=50.0, incl_deg=75.0, fov_deg=25.0, width=width, height=rows)
    tracer.set_launch_config()
    inner = 12.0 if spin < 0.0 else 6.0  # a torus of retrograde orbits lies outside their larger last stable one
    tracer.set_shading(relsim.shading(hydro_model=2, tonemapping_mode=1, torus_inner_radius=inner, torus_center_radius=2 * inner))
    try:
        frame = tracer.dispatch(relsim.make_camera(**kw), fields=["status", "r", "phi"])
        first, count = rows // 2 - 20, 40
        part = tracer.dispatch(relsim.make_camera(row_offset=first, row_count=count, **kw), fields=["status", "r", "phi"])
    finally:
        tracer.set_shading(None)
    for f in frame:
        assert part[f].tobytes() == frame[f][first * width:(first + count) * width].tobytes(), f
    assert np.any(part["pixels"]["r"] > 0.0)
