"""The march's packed CDF (two borders per instruction) follows the scalar erf's
branches: frames whose bins lie in the series' range only, across the branch
points, and mostly beyond saturation give the oracle's image bit for bit (the
oracle evaluates every border with its own scalar erf)."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from oracle import oracle as O
from test_gpu_parity import run_vm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,scale_range,extent", [(1, (0.3, 0.3), 0.01), (40, (0.2, 0.3), 0.3), (400, (0.003, 0.2), 0.8)])
def test_image_bits(cuda, n, scale_range, extent):
    sc = S.make_scene(n, seed=n, extent=extent, scale_range=scale_range)
    cam = S.make_camera(40, 24)
    ref = O.vm_forward(sc, cam, dtype=np.float32)
    cache, _ = run_vm(sc, cam, cuda, torch.float32)
    np.testing.assert_array_equal(cache[0].cpu().numpy(), ref["fb"])
    np.testing.assert_array_equal(cache[12].cpu().numpy(), ref["remaining_transparency"])
