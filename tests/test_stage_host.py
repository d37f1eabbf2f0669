"""The one-copy read-back of small host dispatches (csrc/rt_stage.h, compiled here for
the host): where the outputs lie, and which dispatches copy field by field instead:
banded ones, large ones, and any for which a buffer cannot be had."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import relsim

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SIZES = [np.dtype(dt).itemsize for _, dt in relsim.RAY_FIELDS]
ALL = (1 << len(SIZES)) - 1


@pytest.fixture(scope="module")
def stage(tmp_path_factory):
    out = tmp_path_factory.mktemp("stage") / "libstage_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "relativity-simulator_b200", "csrc"), os.path.join(HERE, "stage", "stage_host.cpp"),
                    "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    L.host_stage.argtypes = [ctypes.c_uint, ctypes.c_int, ctypes.c_long, ctypes.c_int, ctypes.c_void_p]
    L.host_stage.restype = ctypes.c_long

    def run(mask, pixels, n, fail=0):
        at = np.empty(len(SIZES) + 1, dtype=np.int64)
        return L.host_stage(mask, int(pixels), n, fail, at.ctypes.data), at

    return run


@pytest.mark.parametrize("mask", [1, 1 << 17, 0b1000010000, ALL])
@pytest.mark.parametrize("pixels", [False, True])
@pytest.mark.parametrize("n", [1, 63, 4096, 20001])
def test_outputs_lie_apart(stage, mask, pixels, n):
    total, at = stage(mask, pixels, n)
    size = [s if mask >> f & 1 else 0 for f, s in enumerate(SIZES)] + [relsim.PIXEL_DTYPE.itemsize if pixels else 0]
    spans = sorted((a, a + n * s) for a, s in zip(at, size) if s)
    assert all((a >= 0) == (s > 0) for a, s in zip(at, size))
    assert all(a % 256 == 0 for a, _ in spans) and spans[-1][1] <= total <= 4 << 20
    assert all(b <= c for (_, b), (c, _) in zip(spans, spans[1:]))


@pytest.mark.parametrize("mask,pixels,n,staged", [
    (1, False, (1 << 20) - 1, True), (1, False, 1 << 20, False), (1, False, (1 << 20) + 1, False),
    (1 << 4, False, 1 << 19, True), (1 << 4, False, (1 << 19) + 1, False), (0, False, 64, False),
    (0, True, 64, True)])
def test_large_and_banded_dispatches_copy_by_field(stage, mask, pixels, n, staged):
    total, at = stage(mask, pixels, n)
    assert (total > 0) == staged and staged == bool(np.any(at >= 0))


@pytest.mark.parametrize("fail", [1, 2])
def test_without_memory_fields_are_copied_by_themselves(stage, fail):
    total, at = stage(ALL, True, 4096, fail)
    assert total == 0 and np.all(at == -1)
