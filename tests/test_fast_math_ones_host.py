"""The arguments on which Markstein's correction of a reciprocal hangs (csrc/rt_fast_math.h):
a significand of all ones, which tests/test_fast_math_host.py leaves out and whose
reciprocal may be one ulp low, and the 32 significands B with B M = 2^106 - 2, M odd,
whose reciprocals lie closest above a midpoint of two doubles."""
import numpy as np
from test_fast_math_host import refine  # noqa: F401

CLOSE = np.array([
    0x1024a3bd98da02, 0x10699d36aec84e, 0x109107683ee29e, 0x110af85de838ce, 0x11d3799c32581e, 0x11f98ea5d9b262,
    0x12bf5907e316d2, 0x12e93952a2ed6e, 0x130a0dd90e13a2, 0x134d8fe343ef42, 0x13a324a526d5ee, 0x14a6fb45f5d782,
    0x14cad5a5fa03ee, 0x155f2490c86132, 0x163baaac17d1e2, 0x163dd0554d0122, 0x17641c46f799ee, 0x178cb7d5d6e322,
    0x17f52093014f0e, 0x184a12efef626e, 0x199e1b447e99c2, 0x19f142d24e1352, 0x1a0b8ffffcbe8e, 0x1a6f41dab98cb2,
    0x1b227794e85702, 0x1bea3278b789d2, 0x1d5b9032f086be, 0x1da210daeb138e, 0x1de441d5331432, 0x1e20adbc4078a2,
    0x1e756f08df1792, 0x1ef7930608393e], dtype=np.uint64)


def close_to_midpoints(lo, hi):
    """Those significands at every exponent from lo to hi."""
    e = np.arange(lo, hi + 1).astype(np.uint64) + np.uint64(1023)
    return ((e[:, None] << np.uint64(52)) | (CLOSE[None, :] & np.uint64((1 << 52) - 1))).ravel().view(np.float64)


def test_close_significands_lie_above_midpoints():
    for b in CLOSE.tolist():
        m, rest = divmod(2 ** 106 - 2, b)
        assert rest == 0 and m % 2 == 1 and 2 ** 52 <= b < 2 ** 53 <= m < 2 ** 54


def test_reciprocals_next_to_midpoints(refine):  # noqa: F811
    v = close_to_midpoints(-20, 20)
    for off in np.linspace(-1.0, 1.0, 401) * 2.0 ** -19:
        np.testing.assert_array_equal(refine(v, (1.0 / v) * (1.0 + off), 1.0 / np.sqrt(v))[0], 1.0 / v)


def test_reciprocal_of_all_ones_within_an_ulp(refine):  # noqa: F811
    v = np.nextafter(2.0 ** np.arange(-890, 1010, dtype=np.float64), 0.0)
    for off in np.linspace(-1.0, 1.0, 41) * 2.0 ** -19:
        rcp, root = refine(v, (1.0 / v) * (1.0 + off), (1.0 / np.sqrt(v)) * (1.0 + off))
        assert np.all((rcp == 1.0 / v) | (rcp == np.nextafter(1.0 / v, 0.0)))
        np.testing.assert_array_equal(root, np.sqrt(v))
