"""The packed splat backward (two pixels per lane) at its own edges, against the
oracle: frames whose 8x8 quarters and pixel pairs lie partly outside, and
upstream gradients past the packed walk's magnitudes, which take the guarded
walk.  A non-finite gradient at one pixel reaches only the Gaussians of that
pixel.  Bar as in test_gpu_parity: 1e-3 per element."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S, splat
from oracle import oracle as O
from test_gpu_parity import GRAD_TOL, grad_err, run_splat

pytestmark = pytest.mark.gpu

GRAD_NAMES = ("sh", "weights", "centroids", "scales", "rotations")


@pytest.mark.parametrize("w,h,scale", [(64, 48, 1.0), (57, 37, 1.0), (9, 4, 1.0), (8, 5, 1.0), (57, 37, 1e20)])
def test_gradients_match_oracle(cuda, w, h, scale):
    sc = S.make_scene(1500, seed=w, sh_degree=1)
    cam = S.make_camera(w, h)
    G = (np.random.default_rng(h).normal(size=(3, h, w)) * scale).astype(np.float32)
    ref = O.splat_forward(sc, cam)
    gref = O.splat_backward(sc, cam, ref, G)
    _, frame, ts = run_splat(sc, cam, cuda)
    grads = splat.splat_backward(frame, torch.tensor(G, device=cuda), *ts)
    for name, g in zip(GRAD_NAMES, grads):
        e = grad_err(g.cpu().numpy().reshape(gref[name].shape), gref[name])
        assert e <= GRAD_TOL, (name, e)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_non_finite_pixel_stays_with_its_gaussians(cuda, value):
    sc = S.make_scene(1500, seed=3)
    cam = S.make_camera(64, 48)
    G = np.random.default_rng(1).normal(size=(3, 48, 64)).astype(np.float32)
    _, frame, ts = run_splat(sc, cam, cuda)
    v = {k: t.cpu().numpy() for k, t in frame.views().items()}
    x, y = 21, 30
    # the Gaussians whose alpha reaches 1/255 at the pixel (with a margin on the cutoff)
    d = np.array([x, y], dtype=np.float64) - v["points_xy_image"]
    co = v["conic_opacity"].astype(np.float64)
    q = co[:, 0] * d[:, 0] ** 2 + 2 * co[:, 1] * d[:, 0] * d[:, 1] + co[:, 2] * d[:, 1] ** 2
    reach = (v["tiles_touched"] > 0) & (co[:, 3] * np.exp(-0.5 * q) > 0.99 / 255)
    assert 0 < reach.sum() < 1000
    clean = splat.splat_backward(frame, torch.tensor(G, device=cuda), *ts)
    G[:, y, x] = value
    dirty = splat.splat_backward(frame, torch.tensor(G, device=cuda), *ts)
    for name, a, b in zip(GRAD_NAMES, clean, dirty):
        a, b = (t.cpu().numpy().reshape(sc.n, -1)[~reach] for t in (a, b))
        assert np.isfinite(b).all(), name
        assert grad_err(b, a) <= GRAD_TOL, name
    assert not np.isfinite(dirty[0].cpu().numpy().reshape(sc.n, -1)[reach]).all()
