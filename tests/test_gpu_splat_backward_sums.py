"""The sums of the splat backward: a splat's partials are added in float over 32
pixels at most (the even or the odd columns of an 8x8 quarter), and in double from
there on."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S, splat
from test_gpu_parity import cam_tensors, to_dev

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
