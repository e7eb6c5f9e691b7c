"""The SH gradient rows of the splat backward at the edges of a warp's copy:
counts around 32 and 128, every coefficient count, and a batch in which scenes of
different coefficient counts meet inside a warp, against the oracle and against
the scenes on their own."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S, splat
from differentiable_gaussian_mixture_renderer_b200.batch import BatchRenderer
from differentiable_gaussian_mixture_renderer_b200.serving import GaussianScene
from oracle import oracle as O
from test_gpu_parity import GRAD_TOL, grad_err, run_splat

pytestmark = pytest.mark.gpu

GRAD_NAMES = ("sh", "weights", "centroids", "scales", "rotations")


@pytest.mark.parametrize("degree", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129])
def test_rows_match_oracle(cuda, n, degree):
    sc = S.make_scene(n, seed=n + degree, sh_degree=degree, extent=0.6, scale_range=(0.02, 0.2))
    cam = S.make_camera(48, 40)
    G = np.random.default_rng(n).normal(size=(3, 40, 48)).astype(np.float32)
    ref = O.splat_forward(sc, cam)
    gref = O.splat_backward(sc, cam, ref, G)
    _, frame, ts = run_splat(sc, cam, cuda)
    for name, g in zip(GRAD_NAMES, splat.splat_backward(frame, torch.tensor(G, device=cuda), *ts)):
        assert grad_err(g.cpu().numpy().reshape(gref[name].shape), gref[name]) <= GRAD_TOL, name


def test_scenes_that_meet_inside_a_warp(cuda):
    degrees = {"a": (45, 1), "b": (70, 3), "c": (3, 0), "d": (33, 2)}
    host = {k: S.make_scene(n, seed=n, sh_degree=d, extent=0.6, scale_range=(0.02, 0.2)) for k, (n, d) in degrees.items()}
    scenes = {k: GaussianScene.from_numpy(s, cuda) for k, s in host.items()}
    cams = S.random_cameras(5, 48, 40, seed=3)
    views = [("a", cams[0]), ("b", cams[1]), ("c", cams[2]), ("d", cams[3]), ("b", cams[4])]
    r = BatchRenderer(scenes)
    p = r.plan(views, backward=True)
    want = {k: None for k in scenes}
    for (k, cam), g in zip(views, p.grad_framebuffers):
        g.copy_(torch.tensor(np.random.default_rng(cam.width).normal(size=(3, 40, 48)).astype(np.float32)))
        _, frame, ts = run_splat(host[k], cam, cuda)
        got = splat.splat_backward(frame, g, *ts)
        want[k] = got if want[k] is None else [a + b for a, b in zip(want[k], got)]
    r.forward(p)
    r.backward(p)
    torch.cuda.synchronize()
    for k in scenes:
        for name, a, b in zip(GRAD_NAMES, p.grads[k], want[k]):
            err = float((a.reshape(-1) - b.reshape(-1)).abs().max()) / (float(b.abs().max()) + 1e-30)
            assert err <= 1e-5, (k, name, err)
