"""The packed float functions of the kernels are their scalar forms, bit for bit,
for every float of the ranges that they are used on: the reciprocal of 1 - alpha
against the division, the exponential and erf against the scalar functions that
the oracle shares."""
import ctypes as C
import os
import struct
import subprocess

import pytest

from differentiable_gaussian_mixture_renderer_b200 import build as B

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def bits(x):
    return struct.unpack("<I", struct.pack("<f", x))[0]


def device_shim(name, folder):
    """A shared library of tests/kat_shim/<name>.cu, compiled as the kernels are."""
    out = str(folder / (name + ".so"))
    subprocess.run([B.nvcc(), *B.host_compiler(), "-std=c++17", "-O3", *B.ARCH, "-fmad=false", "-prec-div=true", "-prec-sqrt=true",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-I", B.CSRC, "-o", out,
                    os.path.join(HERE, "kat_shim", name + ".cu")], check=True)
    return C.CDLL(out)


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    lib = device_shim("packed_math", tmp_path_factory.mktemp("packed"))
    lib.packed_math_mismatches.restype = C.c_longlong
    lib.packed_math_mismatches.argtypes = [C.c_int, C.c_uint32, C.c_uint32, C.POINTER(C.c_uint32)]
    return lib


@pytest.mark.parametrize("function,lo,hi", [
    (0, bits(0.0099), bits(1.0)),  # reciprocal
    (1, bits(-0.0), bits(-87.0)), (1, bits(0.0), bits(85.0)),  # exponential
    (2, 0, 0xffffffff),  # erf: NaN and infinities among them
])
def test_every_float_of_the_range(cuda, shim, function, lo, hi):
    one = C.c_uint32()
    bad = shim.packed_math_mismatches(function, lo, hi, C.byref(one))
    assert bad == 0, (bad, hex(one.value))


def test_the_comparison_sees_a_difference(cuda, shim):
    """Subnormals are outside the reciprocal's range: it flushes them."""
    one = C.c_uint32()
    assert shim.packed_math_mismatches(0, 1, 1000, C.byref(one)) == 2 * 1000 and 1 <= one.value <= 1000
