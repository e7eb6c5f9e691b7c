"""vol_raster's packed passes where they can go wrong, against the oracle: an
odd last Gaussian of a batch, batches just full, frames of a few Gaussians that
never fill the bins, and ones that fill them and merge."""
import numpy as np
import pytest

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from oracle import oracle as O
from test_gpu_vol_raster import IMAGE_TOL, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extent,scales", [(1, 0.01, (0.1, 0.2)), (2, 0.05, (0.1, 0.2)), (31, 0.2, (0.1, 0.3)), (33, 0.2, (0.1, 0.3)),
                                             (64, 0.5, (0.05, 0.3)), (65, 0.5, (0.02, 0.3)), (600, 0.4, (0.004, 0.1))])
def test_small_frames_match_oracle(cuda, n, extent, scales):
    sc = S.make_scene(n, seed=n, extent=extent, scale_range=scales)
    cam = S.make_camera(37, 21, eye=(0.1, 0.0, -1.5))
    ref = O.vr_forward(sc, cam, bg=np.array((0.1, 0.2, 0.3), np.float32))
    fb = _run(sc, cam, (0.1, 0.2, 0.3)).cpu().numpy()
    assert np.isfinite(fb).all()
    assert float(np.abs(fb - ref["fb"]).max()) <= IMAGE_TOL
