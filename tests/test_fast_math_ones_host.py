"""The one kind of argument that tests/test_fast_math_host.py leaves out: a significand
of all ones, whose reciprocal Markstein's correction may leave one ulp low
(csrc/rt_fast_math.h)."""
import numpy as np
from test_fast_math_host import refine  # noqa: F401


def test_reciprocal_of_all_ones_within_an_ulp(refine):  # noqa: F811
    v = np.nextafter(2.0 ** np.arange(-890, 1010, dtype=np.float64), 0.0)
    for off in np.linspace(-1.0, 1.0, 41) * 2.0 ** -19:
        rcp, root = refine(v, (1.0 / v) * (1.0 + off), (1.0 / np.sqrt(v)) * (1.0 + off))
        assert np.all((rcp == 1.0 / v) | (rcp == np.nextafter(1.0 / v, 0.0)))
        np.testing.assert_array_equal(root, np.sqrt(v))
