"""The blend of two pixels per lane against the blend of a pixel per thread (the
16x16 blocks a batch may choose), bit for bit: frames whose quarters and pixel
pairs lie partly outside, and records that the packed walk hands to its guarded
copy -- non-finite or huge colours and opacities, splats far from the frame."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from differentiable_gaussian_mixture_renderer_b200.batch import BatchRenderer
from differentiable_gaussian_mixture_renderer_b200.serving import GaussianScene

pytestmark = pytest.mark.gpu


def images(scene, cams, block, cuda):
    r = BatchRenderer({0: GaussianScene.from_numpy(scene, cuda)}, blend_block=block)
    p = r.plan([(0, c) for c in cams])
    r.forward(p)
    torch.cuda.synchronize()
    assert not p.overflowed()
    return [fb.cpu().numpy() for fb in p.framebuffers]


@pytest.mark.parametrize("kind", ["plain", "colour", "opacity", "scales"])
def test_quarters_are_the_tiles(cuda, kind):
    sc = S.make_scene(4000, seed=11, sh_degree=1)
    rng = np.random.default_rng(12)
    odd = rng.choice(sc.n, size=60, replace=False)
    if kind == "colour":
        sc.sh[odd, 0, 0] = rng.choice([np.inf, -np.inf, np.nan, 1e30, 3e38], size=60)
    elif kind == "opacity":
        sc.weights[odd] = rng.choice([np.inf, np.nan, 1e25, 3e38, -1.0, 0.0], size=60)
    elif kind == "scales":
        sc.scales[odd] *= rng.choice([1e-6, 30.0, 1e4], size=(60, 1))
    cams = [S.make_camera(w, h, eye=(0.2, 0.1, -2.0)) for w, h in ((64, 48), (57, 37), (9, 4), (8, 5), (16, 16), (1, 1), (203, 111))]
    for a, b in zip(images(sc, cams, 8, cuda), images(sc, cams, 16, cuda)):
        np.testing.assert_array_equal(a, b)
        assert np.isfinite(a).any()
