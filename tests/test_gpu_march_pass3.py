"""The march backward's last pass takes which entries lie on the bins from the
pass before it, for a ray's first 32 batches of 32 entries, and tests later
batches again: rays with usable entries on both sides of that line (float32
keeps 1024 packed, float64 512 and then reads the rest of the tile's list),
against the oracle.  Bars as in test_gpu_parity.
"""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from test_gpu_march_ray_list import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dtype", [(31, torch.float32), (65, torch.float32), (1024, torch.float32), (1057, torch.float32),
                                     (1024, torch.float64), (1060, torch.float64)])
def test_entries_on_the_bins(cuda, n, dtype):
    """A loose cluster (the opaque one's gradients hang on the order of its sums)."""
    sc = S.make_scene(n, seed=n, extent=0.1, scale_range=(0.08, 0.1))
    sc.weights = np.random.default_rng(n).uniform(0.01, 0.05, size=n).astype(np.float32)
    check(sc, S.make_camera(18, 17, eye=(0.1, 0.05, -0.9)), cuda, dtype)
