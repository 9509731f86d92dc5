"""The warp's many-sums exchange (deb_warp_sums.cuh), its lanes emulated on the host.

Each sum must be stored by one lane and no other: lanes that store different
values to one address in one instruction leave open which of them stays.
The inputs are integers, so the sums are exact in any order.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")
_SRC = os.path.join(_DIR, "warp_sums_harness.cpp")
_LIB = os.path.join(_DIR, "_build", "libwarp_sums_harness.so")


@pytest.fixture(scope="module")
def lib():
    os.makedirs(os.path.dirname(_LIB), exist_ok=True)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-pthread", "-o", _LIB, _SRC])
    return ctypes.CDLL(_LIB)


@pytest.mark.parametrize("n", range(1, 21))
def test_each_sum_is_stored_by_one_lane(lib, n):
    x = np.random.default_rng(n).integers(1, 1 << 20, size=(32, n)).astype(np.float64)
    out = np.full((32, n), np.nan)
    p = ctypes.POINTER(ctypes.c_double)
    assert lib.h_warp_sums(n, x.ctypes.data_as(p), out.ctypes.data_as(p)) == 0
    stored = ~np.isnan(out)
    np.testing.assert_array_equal(stored.sum(axis=0), 1)
    np.testing.assert_array_equal(np.nansum(out, axis=0), x.sum(axis=0))
