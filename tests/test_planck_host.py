"""The blackbody colour's table (csrc/rt_planck.h, compiled here for the host)
against the spectral sum it replaces: over the table's temperatures, at its ends,
beyond its upper clamp and on both sides of the borders between pieces.  Bar
1e-13 relative (interpolation remainder below 1e-15; the sum's 33 terms and the
interpolant's coefficients each carry a few dozen roundings)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "relativity-simulator_b200", "csrc")


def _lobe(x, alpha, mu, s1, s2):
    return alpha * np.exp(-0.5 * ((x - mu) / np.where(x < mu, s1, s2)) ** 2)


@pytest.mark.parametrize("where", ["spread", "ends", "borders"])
def test_table_matches_the_sum(tmp_path, where):
    so = tmp_path / "libplanck_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
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
    if where == "spread":
        t = np.exp(np.random.default_rng(1).uniform(np.log(500.0), np.log(4e5), 20000))
    elif where == "ends":
        t = np.array([500.0, np.nextafter(500.0, 1e3), 4e5, np.nextafter(4e5, 0.0), 5e5, 1e9])
    else:
        s = 1 / 4e5 + np.arange(257) * (1 / 500.0 - 1 / 4e5) / 256
        t = np.concatenate([1 / (s * (1 + d)) for d in (-1e-15, 0.0, 1e-15)])
        t = t[t >= 500.0]
    got = np.empty((2, t.size, 3))
    t = np.ascontiguousarray(t)
    L.host_planck(lam.ctypes.data, w.ctypes.data, t.ctypes.data, t.size, got[0].ctypes.data, got[1].ctypes.data)
    rel = np.abs(got[1] / got[0] - 1.0)
    print("max relative difference", rel.max())
    assert rel.max() < 1e-13
