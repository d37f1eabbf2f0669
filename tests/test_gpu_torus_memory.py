"""The torus's scratch memory is given back when a handle's shading is switched off, and
taken again, for the same frame, when it is switched on."""
import pytest

import relsim

pytestmark = pytest.mark.gpu


def test_switching_shading_off_gives_the_memory_back():
    import torch

    def used():
        free, total = torch.cuda.mem_get_info()
        return (total - free) / 2 ** 20

    cam = relsim.make_camera(spin=0.9, r_obs=50.0, incl_deg=75.0, fov_deg=25.0, width=320, height=180)
    torus = relsim.shading(hydro_model=2, tonemapping_mode=1, torus_inner_radius=6.0, torus_center_radius=10.0)
    torch.zeros(1, device="cuda")
    with relsim.Tracer(0) as tr:
        tr.dispatch(cam, fields=[])  # unshaded: its buffers and the kernels are there
        before = used()
        tr.set_shading(torus)
        first = tr.dispatch(cam, fields=[])["pixels"]
        shaded = used()
        tr.set_shading(None)
        after = used()
        tr.set_shading(torus)
        again = tr.dispatch(cam, fields=[])["pixels"]
    # five pages of 1,544 bytes a ray, and 300 bytes of other shading scratch; 2 MB granules
    pool = 320 * 180 * 5 * 1544 / 2 ** 20
    assert shaded - before > 0.95 * pool
    assert after - before < 0.1 * pool
    assert first.tobytes() == again.tobytes()
