"""A batch whose scenes hold no Gaussian, and one where such a scene stands beside
another: images of the background alone, no record read."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from differentiable_gaussian_mixture_renderer_b200.batch import BatchRenderer
from differentiable_gaussian_mixture_renderer_b200.serving import GaussianScene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [8, 16])
@pytest.mark.parametrize("n_other", [None, 300])
def test_scenes_without_gaussians_draw_the_background(cuda, block, n_other):
    scenes = {0: GaussianScene.from_numpy(S.make_scene(0, seed=1), cuda)}
    if n_other:
        scenes[1] = GaussianScene.from_numpy(S.make_scene(n_other, seed=2), cuda)
    r = BatchRenderer(scenes, blend_block=block)
    cams = [S.make_camera(40, 32), S.make_camera(57, 37)]
    p = r.plan([(k, c) for c in cams for k in scenes])
    r.forward(p)
    torch.cuda.synchronize()
    assert not p.overflowed()
    for (k, cam), fb in zip([(k, c) for c in cams for k in scenes], p.framebuffers):
        assert (np.abs(fb.cpu().numpy()).max() == 0) == (k == 0)
