"""The step loops' FP64 reciprocal and square root (csrc/rt_fast_math.h, compiled
here for the host) from seeds as coarse as the hardware's: equal to IEEE 1 / v
and sqrt(v) bit for bit over their range, NaN for arguments without a finite
seed.  (A significand of all ones, where Markstein's correction of a reciprocal
may be one ulp off, is left out.)"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "relativity-simulator_b200", "csrc")


@pytest.fixture(scope="module")
def refine(tmp_path_factory):
    out = tmp_path_factory.mktemp("fast_math") / "libfast_math_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "fast_math", "fast_math_host.cpp"), "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    p = ctypes.c_void_p
    L.host_refine.argtypes = [p, p, p, ctypes.c_long, p, p]

    def run(v, s_rcp, s_rsqrt):
        a = [np.ascontiguousarray(x, dtype=np.float64) for x in (v, s_rcp, s_rsqrt)]
        out = np.empty((2, a[0].size))
        L.host_refine(*(x.ctypes.data for x in a), a[0].size, out[0].ctypes.data, out[1].ctypes.data)
        return out

    return run


@pytest.mark.parametrize("lo,hi", [(-40, 40), (-900, -860), (960, 1019), (-900, 1019)])
def test_refined_values_are_correctly_rounded(refine, lo, hi):
    rng = np.random.default_rng(2000 + hi)
    n = 400_000
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    m[:2000] = np.arange(2000, dtype=np.uint64)                            # just above a power of two
    m[2000:4000] = (1 << 52) - 2 - np.arange(2000, dtype=np.uint64)        # just below one
    e = rng.integers(lo, hi + 1, n).astype(np.uint64) + np.uint64(1023)
    v = ((e << np.uint64(52)) | m).view(np.float64)
    off = 1.0 + rng.uniform(-1.0, 1.0, n) * 2.0 ** -19
    rcp, root = refine(v, (1.0 / v) * off, (1.0 / np.sqrt(v)) * off)
    np.testing.assert_array_equal(rcp, 1.0 / v)
    np.testing.assert_array_equal(root, np.sqrt(v))


def test_arguments_without_a_finite_seed_give_nan(refine):
    """Hardware seeds: infinite for zero and (flushed) subnormals, zero for infinity, NaN otherwise."""
    inf, nan = np.inf, np.nan
    v = [0.0, 5e-324, 1e-310, inf, nan]
    s = [inf, inf, inf, 0.0, nan]
    rcp, root = refine(v, s, s)
    assert np.all(np.isnan(rcp)) and np.all(np.isnan(root))
    _, root = refine([-1.0, -inf], [1.0, 0.0], [nan, nan])
    assert np.all(np.isnan(root))
