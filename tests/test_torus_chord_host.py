"""One chord's light through the torus (fm_chord of csrc/rt_shade.cuh, on the host and on
the device) against the reference's chord integral in extended precision, beside that
integral in double (tests/torus/chord_host.cu): over tori of several spins and adiabatic
indices the library's light, opacity and redshift are on average no further off than the
double integral's.  (The averages are of a sample of chords, and two roundings of the same
quality differ in them by chance: the bar is three standard errors of the mean of the
chords' differences.)"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
from test_planck_host import _lobe

import relsim

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
N = 4000


@pytest.fixture(scope="module")
def chords_lib(tmp_path_factory):
    import build

    if np.finfo(np.longdouble).eps > 2e-19:
        pytest.skip("no extended precision")
    out = tmp_path_factory.mktemp("chord") / "libchord_host.so"
    subprocess.run([build.nvcc(), *build.GENCODE, "-O2", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC,-mfma,-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "relativity-simulator_b200", "csrc"), os.path.join(HERE, "torus", "chord_host.cu"),
                    "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    d, p = ctypes.c_double, ctypes.c_void_p
    L.chords.argtypes = [ctypes.c_int, d, d, p, p, p, ctypes.c_long, p, p]
    L.chords.restype = ctypes.c_long
    return L


def _spectrum():
    nm = 380.0 + 12.5 * np.arange(33)
    trap = np.where((np.arange(33) == 0) | (np.arange(33) == 32), 0.5, 1.0)
    w = np.stack([
        trap * (_lobe(nm, 1.056, 599.8, 37.9, 31.0) + _lobe(nm, 0.362, 442.0, 16.0, 26.7) - _lobe(nm, 0.065, 501.1, 20.4, 26.2)),
        trap * (_lobe(nm, 0.821, 568.8, 46.9, 40.5) + _lobe(nm, 0.286, 530.9, 16.3, 31.1)),
        trap * (_lobe(nm, 1.217, 437.0, 11.8, 36.0) + _lobe(nm, 0.681, 459.0, 26.0, 13.8))], axis=1)
    return np.ascontiguousarray(nm * 1e-3), np.ascontiguousarray(w)


@pytest.mark.parametrize("where", ["host", pytest.param("device", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("gamma", [1.01, 1.05, 4.0 / 3.0, 5.0 / 3.0])
@pytest.mark.parametrize("spin", [0.0, 0.5, 0.9, 0.998])
def test_chords_are_no_further_off_than_the_double_integral(chords_lib, spin, gamma, where):
    lam, w = _spectrum()
    disk = np.frombuffer(bytes(relsim.shading().disk), dtype=np.float32).copy()
    disk[3], disk[4], disk[7], disk[9], disk[28] = 23796.0, 1200.0, 5.32, 1.0, 0.0  # peak, floor, beaming, saturation
    kelvin = 14387.76877 / (lam * 23796.0)
    disk[28] = ((1.0 / (lam ** 5 * np.expm1(kelvin))) * w[:, 1]).sum()  # the reference luminance
    g = np.random.default_rng(int(1000 * spin) + int(100 * gamma))
    r, th = g.uniform(5.0, 40.0, N), np.arccos(g.uniform(-0.6, 0.6, N))
    ph, step = g.uniform(-np.pi, np.pi, N), np.exp(g.uniform(np.log(0.05), np.log(8.0), N))
    start = np.stack([r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), r * np.cos(th)], axis=1)
    way = g.normal(size=(N, 3))
    end = start + way * (step / np.linalg.norm(way, axis=1))[:, None]
    chords = np.ascontiguousarray(np.concatenate([start, end, g.uniform(-8.0, 8.0, (N, 1))], axis=1))
    err = np.empty((2, 5, N))
    odd = chords_lib.chords(where == "device", spin, gamma, lam.ctypes.data, w.ctypes.data, disk.ctypes.data, N, chords.ctypes.data,
                                 err.ctypes.data)
    assert odd == 0
    for k, name in enumerate(["red", "green", "blue", "opacity", "redshift"]):
        ours, plain = err[:, k, err[0, k] >= 0.0]
        assert ours.size > N // 16
        print(f"  {name:9s} mean {ours.mean():.2e} / {plain.mean():.2e}  max {ours.max():.2e} / {plain.max():.2e}")
        more = ours - plain
        assert more.mean() <= 3.0 * more.std() / np.sqrt(more.size), name
