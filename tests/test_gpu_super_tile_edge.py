"""The largest frame whose super-tiles are planned from one sort pass, 255 of them,
and 256, which take two: their ids have a ninth bit, the count's own.  (The check
of test_gpu_binning_sizes, whose frames of 256 and 289 super-tiles both take two.)"""
import pytest

import test_gpu_binning_sizes as sizes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h", [(5_000, 17 * 128, 15 * 128), (5_000, 17 * 128 - 15, 15 * 128 - 1), (5_000, 16 * 128, 16 * 128)])
def test_binning_on_both_sides_of_one_sort_pass(cuda, n, w, h):
    sizes.test_binning_is_its_definition(cuda, n, w, h, 1.5)
