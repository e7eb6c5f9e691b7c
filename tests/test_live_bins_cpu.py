"""The bins that the march's backward leaves out as too far from a Gaussian on
the ray: none of them reaches the mass test of 1e-5, for every mass that the
march accepts (1/255 to 1000)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    out = str(tmp_path_factory.mktemp("live") / "live.so")
    subprocess.run([cxx, "-O2", "-march=x86-64-v3", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", out,
                    os.path.join(HERE, "kat_shim", "live_bins.cpp")], check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("is_double", [0, 1])
def test_bins_left_out_fail_the_mass_test(lib, is_double):
    mor = np.concatenate([np.geomspace(1.0 / 255.0, 1000.0, 400), [9.98, 9.99, 10.0]])
    limit, largest = np.empty_like(mor), np.empty_like(mor)
    ptr = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
    lib.live_bins(is_double, ptr(mor), C.c_long(len(mor)), C.c_long(50_000), ptr(limit), ptr(largest))
    assert np.all(largest < 1e-5)
    cut = 5.0 if is_double else 3.92
    assert np.all((limit >= 2.0) & (limit <= cut + 1e-6))
    assert np.all(limit[mor < 1.0] < 3.2)
