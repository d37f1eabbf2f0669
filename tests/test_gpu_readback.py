"""Host dispatches about the size from which they are traced and copied in bands (2^20
rays): every four-byte record field asked for alone holds the bytes of a device
dispatch, also after a small dispatch whose outputs came back in one copy."""
import numpy as np
import pytest

import relsim
from cameras import config_cam

pytestmark = pytest.mark.gpu
FIELDS = ["status", "flags", "steps_accepted", "steps_rejected", "body"]
KINDS = {
    "fp64": dict(precision=relsim.PRECISION_FP64),
    "mixed": dict(precision=relsim.PRECISION_MIXED),
    "boyer_lindquist": dict(metric_form=relsim.METRIC_BOYER_LINDQUIST, charge=0.3),
}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows", [1023, 1024, 1025])
def test_one_field_alone(tracer, kind, rows):
    import torch

    tracer.set_launch_config()
    cam = config_cam("c2", width=1024, height=rows, rtol=1e-6, atol=1e-6, **KINDS[kind])
    n = 1024 * rows
    dev = {f: torch.full((n,), -1, dtype=torch.int32, device="cuda") for f in FIELDS}
    ro = relsim.RayOut()
    for f, t in dev.items():
        setattr(ro, f, t.data_ptr())
    torch.cuda.synchronize()
    tracer.dispatch_device(cam, ro, None, n)
    tracer.synchronize()
    for f in FIELDS:
        tracer.dispatch(config_cam("c1", width=64, height=64), fields=[f], pixels=False)
        got = tracer.dispatch(cam, fields=[f], pixels=False)[f]
        np.testing.assert_array_equal(got, dev[f].cpu().numpy().view(np.uint32), err_msg=f)
