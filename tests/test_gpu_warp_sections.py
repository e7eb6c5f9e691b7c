"""The march's section insertion by a whole warp -- the device code itself --
against SectionSet::put, which the reference's known answers pin: the same sets bit
for bit after every insertion of random sequences (with equal ends and steps; in
the odd ones also unbounded and empty sections and NaN steps)."""
import ctypes as C

import pytest

from test_gpu_packed_math import device_shim

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    lib = device_shim("warp_sections", tmp_path_factory.mktemp("sections"))
    lib.warp_sections.argtypes = [C.c_int, C.c_int, C.c_uint32, C.c_int, C.POINTER(C.c_ulonglong)]
    return lib


@pytest.mark.parametrize("is_double", [0, 1])
@pytest.mark.parametrize("odd", [0, 1])
def test_warp_insertions_are_put(cuda, shim, is_double, odd):
    got = (C.c_ulonglong * 5)()
    assert shim.warp_sections(is_double, odd, 3 + odd, 40_000, got) == 0
    puts, covered, pieces, full, bad = got
    assert puts > 1_000_000 and full > 10_000 and (covered > 10_000) != bool(odd) and (pieces > 10_000) == bool(odd)
    assert bad == 0
