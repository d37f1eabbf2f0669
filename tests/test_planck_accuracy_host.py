"""The blackbody colour's table (csrc/rt_planck.h, compiled here for the host) and the
spectral sum it stands for, both against the sum in extended precision.  The table has
to be no further off than the sum, at its worst and on average, and within 8e-16: the
interpolation remainder (below 4e-16), the rounding of the leading coefficient, of the
last fused step and of the product with T (1.1e-16 each), and 5e-17 for the terms below."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
from test_planck_host import _lobe

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "relativity-simulator_b200", "csrc")


def test_table_is_no_further_off_than_the_sum(tmp_path):
    if np.finfo(np.longdouble).eps > 2e-19:
        pytest.skip("no extended precision")
    so = tmp_path / "libplanck_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "fast_math", "planck_host.cpp"), "-o", str(so)], check=True)
    L = ctypes.CDLL(str(so))
    p = ctypes.c_void_p
    L.host_planck.argtypes = [p, p, p, ctypes.c_long, p, p]
    nm = 380.0 + 12.5 * np.arange(33)
    trap = np.where((np.arange(33) == 0) | (np.arange(33) == 32), 0.5, 1.0)
    w = np.ascontiguousarray(np.stack([
        trap * (_lobe(nm, 1.056, 599.8, 37.9, 31.0) + _lobe(nm, 0.362, 442.0, 16.0, 26.7) - _lobe(nm, 0.065, 501.1, 20.4, 26.2)),
        trap * (_lobe(nm, 0.821, 568.8, 46.9, 40.5) + _lobe(nm, 0.286, 530.9, 16.3, 31.1)),
        trap * (_lobe(nm, 1.217, 437.0, 11.8, 36.0) + _lobe(nm, 0.681, 459.0, 26.0, 13.8))], axis=1))
    lam = nm * 1e-3
    k = np.arange(1, 263)
    t = np.concatenate([np.exp(np.random.default_rng(3).uniform(np.log(500.0), np.log(4e5), 60000)),
                        [500.0, np.nextafter(500.0, 1e3), 4e5, np.nextafter(4e5, 0.0)],
                        131072.0 / k, np.nextafter(131072.0 / k, 0.0), np.nextafter(131072.0 / k, 1e9)])  # borders
    t = np.ascontiguousarray(t[(t >= 500.0) & (t <= 4e5)])
    got = np.empty((2, t.size, 3))
    L.host_planck(lam.ctypes.data, w.ctypes.data, t.ctypes.data, t.size, got[0].ctypes.data, got[1].ctypes.data)
    X = np.longdouble
    l = lam.astype(X)
    e = X(14387.76877) / (l[None, :] * t.astype(X)[:, None])
    exact = (1 / (l ** 5 * np.expm1(e))) @ w.astype(X)
    err = np.abs(got.astype(X) / exact - 1).astype(np.float64)
    print("sum / table: largest", err[0].max(), err[1].max(), "mean", err[0].mean(), err[1].mean())
    assert err[1].max() <= err[0].max() and err[1].mean() <= err[0].mean()
    assert err[1].max() < 8e-16
