"""The step loops' reciprocal and square root (csrc/rt_fast_math.h) on the device, from
the hardware's own seeds: the bits of the device's IEEE reciprocal and root over the
stated range, one ulp low for the reciprocal of a significand of all ones, and NaN for
the arguments that have no finite seed."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
from test_fast_math_ones_host import close_to_midpoints

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "relativity-simulator_b200", "csrc")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fast(tmp_path_factory):
    import build

    out = tmp_path_factory.mktemp("fast_math") / "libfast_math_device.so"
    subprocess.run([build.nvcc(), *build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "fast_math", "fast_math_device.cu"), "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    L.device_fast.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]

    def run(v):
        v = np.ascontiguousarray(v, dtype=np.float64)
        out = np.empty((4, v.size))
        assert L.device_fast(v.ctypes.data, v.size, out.ctypes.data) == 0
        return out

    return run


def _values(lo, hi, n, seed):
    rng = np.random.default_rng(seed)
    m = rng.integers(0, (1 << 52) - 1, n, dtype=np.uint64)           # all ones left out
    m[:4000] = np.arange(4000, dtype=np.uint64)                      # just above a power of two
    m[4000:8000] = (1 << 52) - 2 - np.arange(4000, dtype=np.uint64)  # just below one
    e = rng.integers(lo, hi + 1, n).astype(np.uint64) + np.uint64(1023)
    return ((e << np.uint64(52)) | m).view(np.float64)


@pytest.mark.parametrize("lo,hi", [(-60, 60), (-900, -860), (960, 1019), (-900, 1019)])
def test_results_are_the_devices_own(fast, lo, hi):
    rcp, root, rcp_rn, root_rn = fast(_values(lo, hi, 1 << 22, 1000 + hi))
    np.testing.assert_array_equal(rcp, rcp_rn)
    np.testing.assert_array_equal(root, root_rn)


def test_reciprocals_next_to_midpoints(fast):
    rcp, root, rcp_rn, root_rn = fast(close_to_midpoints(-900, 1019))
    np.testing.assert_array_equal(rcp, rcp_rn)
    np.testing.assert_array_equal(root, root_rn)


def test_reciprocal_of_all_ones_is_one_ulp_low(fast):
    v = np.nextafter(2.0 ** np.arange(-890, 1010, dtype=np.float64), 0.0)
    rcp, root, rcp_rn, root_rn = fast(v)
    assert np.all((rcp == rcp_rn) | (rcp == np.nextafter(rcp_rn, 0.0)))
    np.testing.assert_array_equal(root, root_rn)


def test_arguments_without_a_finite_seed_give_nan(fast):
    rcp, root, _, _ = fast([0.0, -0.0, 5e-324, 1e-310, np.inf, np.nan])
    assert np.all(np.isnan(rcp)) and np.all(np.isnan(root))
    assert np.all(np.isnan(fast([-1.0, -1e300, -np.inf])[1]))
