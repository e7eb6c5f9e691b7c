"""The sums of the splat backward: a splat's partials are added in float over 32
pixels at most (the even or the odd columns of an 8x8 quarter), and in double from
there on."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S, splat
from oracle import oracle as O
from test_gpu_parity import cam_tensors, run_splat, to_dev

pytestmark = pytest.mark.gpu

ODD, EVEN, BESIDE = (3, 1), (4, 5), (11, 1)  # columns of the first quarter, and a pixel of the second


@pytest.mark.parametrize("out", ["sh", "weights"])
def test_the_columns_of_a_quarter_meet_in_double(cuda, out):
    """The sum over the odd columns is K, over the quarter beside it close to -K, and
    over the even columns less than an ulp of K: it survives."""
    sc = S.make_scene(1, seed=0)
    sc.centroids[:], sc.scales[:], sc.weights[:] = 0.01, 1.0, 0.5
    cam = S.make_camera(16, 16)
    ts = to_dev(sc, cuda)
    view, proj, campos, bg = cam_tensors(cam, cuda)
    _, frame = splat.splat_forward(*ts, view, proj, campos, bg, 16, 16, cam.tan_fovx, cam.tan_fovy, 0, formulation="opacity")
    n = frame.views()["n_contrib"].cpu().numpy()
    assert all(n[y, x] == 1 for x, y in (ODD, EVEN, BESIDE))

    def gradient(at):
        G = torch.zeros((3, 16, 16), device=cuda)
        for (x, y), value in at.items():
            G[0, y, x] = float(np.float32(value))
        return float(splat.splat_backward(frame, G, *ts)[0 if out == "sh" else 1].reshape(-1)[0])

    K = 2.0 ** 30
    k = gradient({ODD: K})
    G3 = -k / gradient({BESIDE: 1.0})
    G2 = 0.37 * 2.0 ** -23 * abs(k) / gradient({EVEN: 1.0})
    rest, low = gradient({ODD: K, BESIDE: G3}), gradient({EVEN: G2})
    got = gradient({ODD: K, BESIDE: G3, EVEN: G2})
    # three results, each of two roundings to float
    assert abs(got - (rest + low)) <= 6 * 2.0 ** -24 * (abs(rest) + abs(low)), (got, rest, low)


def test_the_centre_is_as_close_as_the_other_gradients(cuda):
    """The conic times the offset cancels along a splat's long axis; taken per pixel, in
    float, its error is that of the other per-pixel terms.  2-norm distance from the
    oracle (double sums of the per-pixel floats), mean of six frames: a term has three
    roundings of at most 2^-24 more than the oracle's, sqrt(3) 2^-24 = 1.03e-7 if none
    averaged out."""
    got = []
    for seed in range(6):
        sc = S.make_scene(4000, seed=seed)
        cam = S.make_camera(256, 192)
        G = np.random.default_rng(seed).normal(size=(3, 192, 256)).astype(np.float32)
        ref = O.splat_forward(sc, cam)
        want = O.splat_backward(sc, cam, ref, G)["centroids"].astype(np.float64)
        _, frame, ts = run_splat(sc, cam, cuda)
        g = splat.splat_backward(frame, torch.tensor(G, device=cuda), *ts)[2].cpu().numpy()
        got.append(np.linalg.norm(g - want) / np.linalg.norm(want))
    assert np.mean(got) <= 3 ** 0.5 * 2.0 ** -24, got
