"""The emission of a chunk's pairs, staged and not: rounds of 256 super-tile
entries whose pairs overflow the stage of 4096 (every entry on all 64 tiles of
its super-tile), rounds below it, both in one chunk, and ragged last rounds and
super-tiles.  Checked against the lists' definition, entry for entry."""
import functools

import pytest

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from test_gpu_binning_sizes import test_binning_is_its_definition as check_binning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h,scales", [
    (255, 256, 256, (0.5, 1.0)), (257, 300, 200, (0.5, 1.0)), (1025, 256, 128, (0.5, 1.0)),  # over the stage
    (1500, 200, 136, (0.01, 0.6)),  # around it
    (3000, 128, 128, (0.002, 0.004)),  # about one tile each
])
def test_pairs_are_the_definition(cuda, monkeypatch, n, w, h, scales):
    monkeypatch.setattr(S, "make_scene", functools.partial(S.make_scene, scale_range=scales))
    check_binning(cuda, n, w, h, 1.0)
