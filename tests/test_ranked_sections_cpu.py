"""The marcher's lane-parallel section insertion against SectionSet::put(),
which the reference's known answers pin: the same sets bit for bit after every
insertion of random sequences (with equal ends and steps; in the odd ones also
unbounded and empty sections and NaN steps)."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    out = str(tmp_path_factory.mktemp("ranked") / "ranked.so")
    subprocess.run([cxx, "-O2", "-march=x86-64-v3", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", out,
                    os.path.join(HERE, "kat_shim", "ranked_sections.cpp")], check=True)
    lib = C.CDLL(out)
    lib.ranked_sections.restype = C.c_long
    return lib


@pytest.mark.parametrize("is_double", [0, 1])
@pytest.mark.parametrize("odd", [0, 1])
def test_ranked_insertions_are_put(lib, is_double, odd):
    puts, pieces = C.c_long(), C.c_long()
    bad = lib.ranked_sections(is_double, odd, 3 + odd, 40_000, C.byref(puts), C.byref(pieces))
    assert puts.value > 1_000_000 and (pieces.value > 10_000) == bool(odd)
    assert bad == 0
