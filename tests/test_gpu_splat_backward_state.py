"""What a splat with a non-finite or very large colour leaves behind in the
backward's walk -- the colour behind the next record, on the pixels that it covers
-- stays with those pixels: the gradients of Gaussians that share no pixel with
it are those of the scene with an ordinary colour there."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S, splat
from oracle import oracle as O
from test_gpu_parity import GRAD_TOL, cam_tensors, grad_err, run_splat, to_dev

pytestmark = pytest.mark.gpu

GRAD_NAMES = ("sh", "weights", "centroids", "scales", "rotations")
W, H = 64, 48


def reach_of(v):
    """[N, H, W]: alpha reaches 1/255 there, with a margin on the cutoff."""
    xy, co = v["points_xy_image"].astype(np.float64), v["conic_opacity"].astype(np.float64)
    dx = np.arange(W)[None, None, :] - xy[:, 0, None, None]
    dy = np.arange(H)[None, :, None] - xy[:, 1, None, None]
    q = co[:, 0, None, None] * dx ** 2 + 2 * co[:, 1, None, None] * dx * dy + co[:, 2, None, None] * dy ** 2
    return (v["tiles_touched"] > 0)[:, None, None] & (co[:, 3, None, None] * np.exp(-0.5 * q) > 0.99 / 255)


def deep_splat(v, reach):
    """The Gaussian on the fewest pixels of those that contribute to one, with at
    least 64 entries before it in that tile's list."""
    best = None
    for g in np.flatnonzero(reach.any((1, 2))):
        for y, x in zip(*np.nonzero(reach[g])):
            b, e = v["i_ranges"][(y // 16) * (W // 16) + x // 16]
            at = np.flatnonzero(v["point_list"][b:e] == g)  # empty past the rectangle's tiles
            if at.size and 64 <= at[0] < v["n_contrib"][y, x]:
                n = int(reach[g].sum())
                best = (n, g) if best is None or n < best[0] else best
                break
    return best[1]


@pytest.mark.parametrize("value,scale", [(float("inf"), 1.0), (float("nan"), 1.0), (3e38, 1e6)])
def test_a_huge_colour_stays_with_its_pixels(cuda, value, scale):
    sc = S.make_scene(1500, seed=3)
    cam = S.make_camera(W, H)
    G = torch.tensor(np.random.default_rng(1).normal(size=(3, H, W)) * scale, dtype=torch.float32, device=cuda)
    _, frame, ts = run_splat(sc, cam, cuda)
    v = {k: t.cpu().numpy() for k, t in frame.views().items()}
    reach = reach_of(v)
    bad = deep_splat(v, reach)
    apart = ~(reach & reach[bad]).any((1, 2))
    assert 0 < reach[bad].sum() < 64 and apart.sum() > 1000
    clean = splat.splat_backward(frame, G, *ts)
    sc.sh[bad, 0, 0] = value
    _, frame, ts = run_splat(sc, cam, cuda)
    dirty = splat.splat_backward(frame, G, *ts)
    for name, a, b in zip(GRAD_NAMES, clean, dirty):
        a, b = (t.cpu().numpy().reshape(sc.n, -1)[apart] for t in (a, b))
        assert np.isfinite(b).all(), (name, int((~np.isfinite(b)).any(1).sum()))
        assert grad_err(b, a) <= GRAD_TOL, name


def test_a_huge_product_stays_with_its_pixel(cuda):
    """A splat with an opacity of 1e12 and a colour of 1e15 next to a pixel that it
    does not reach, whose image gradient is 8e17: each is finite, their product is
    not, and none of it belongs to the splat."""
    sc = S.make_scene(1500, seed=3)
    cam = S.make_camera(W, H)
    shs, w, mu, s, q = to_dev(sc, cuda)
    view, proj, campos, bg = cam_tensors(cam, cuda)

    def run():
        _, frame = splat.splat_forward(shs, w, mu, s, q, view, proj, campos, bg, W, H, cam.tan_fovx, cam.tan_fovy, 0, formulation="opacity")
        return frame, {k: t.cpu().numpy() for k, t in frame.views().items()}

    _, v = run()
    # nearest to the middle of an 8x8 quarter, and inside the frame
    xy = v["points_xy_image"]
    mid = np.abs(xy % 8 - 3.5).max(1) + 1e3 * ((v["tiles_touched"] == 0) | (xy < 0).any(1) | (xy > (W - 1, H - 1)).any(1))
    g = int(mid.argmin())
    w[g], shs[g, 0, :], s[g] = 1e12, 1e15, 1e-4
    frame, v = run()
    reach = reach_of(v)[g]
    x0, y0 = (int(c) // 8 * 8 for c in xy[g])
    quarter = reach[y0:y0 + 8, x0:x0 + 8]
    assert quarter.any() and not quarter[0, 0]
    G = torch.tensor(np.random.default_rng(1).normal(size=(3, H, W)), dtype=torch.float32, device=cuda)
    want = splat.splat_backward(frame, G, shs, w, mu, s, q)
    G[:, y0, x0] = 8e17
    got = splat.splat_backward(frame, G, shs, w, mu, s, q)
    for name, a, b in zip(GRAD_NAMES, want, got):
        a, b = a[g].cpu().numpy(), b[g].cpu().numpy()
        assert np.isfinite(a).all() and np.isfinite(b).all(), (name, a, b)
        assert grad_err(b, a) <= GRAD_TOL, name


@pytest.mark.parametrize("weight", [3e38, float("inf"), float("nan")])
def test_a_saturated_splat_has_the_oracles_gradients(cuda, weight):
    """An opacity that overflows (3e38 does, in the Ots formulation) leaves its splat
    saturated on every pixel: its opacity, centre and shape have no gradient."""
    sc = S.make_scene(1500, seed=3)
    sc.weights[100] = weight
    cam = S.make_camera(W, H)
    G = np.random.default_rng(1).normal(size=(3, H, W)).astype(np.float32)
    ref = O.splat_forward(sc, cam)
    assert not np.isfinite(ref["conic_opacity"][100, 3]) and ref["tiles_touched"][100] > 0
    gref = O.splat_backward(sc, cam, ref, G)
    _, frame, ts = run_splat(sc, cam, cuda)
    for name, g in zip(GRAD_NAMES, splat.splat_backward(frame, torch.tensor(G, device=cuda), *ts)):
        g, want = g.cpu().numpy().reshape(gref[name].shape), gref[name]
        fine = np.isfinite(want)
        assert np.isfinite(g[fine]).all(), name
        assert grad_err(g[fine], want[fine]) <= GRAD_TOL, name
