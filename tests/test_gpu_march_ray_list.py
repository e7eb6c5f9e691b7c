"""The march's per-ray lists of usable entries at their limits, against the
oracle: rays with fewer and more usable entries than a warp keeps (1024 in
float32, 512 in float64; the rest of the tile's list is then tested in every
pass), and a tile list longer than the 16-bit offsets reach.

Bars as in test_gpu_parity: bit-exact lists, images within 1e-4 max-abs,
gradients within 1e-3 per element.
"""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import cpp_binding, scene as S
from oracle import oracle as O
from test_gpu_parity import GRAD_TOL, IMAGE_TOL, grad_err, run_vm

pytestmark = pytest.mark.gpu

GRAD_NAMES = ("sh", "weights", "centroids", "scales", "rotations")


def check(sc, cam, dev, dtype):
    npdt = np.float32 if dtype == torch.float32 else np.float64
    ref = O.vm_forward(sc, cam, dtype=npdt)
    cache, ts = run_vm(sc, cam, dev, dtype)
    np.testing.assert_array_equal(cache[11].cpu().numpy(), ref["b_point_list"])
    assert np.abs(cache[0].cpu().numpy() - ref["fb"]).max() <= IMAGE_TOL
    G = np.random.default_rng(5).normal(size=(3, cam.height, cam.width)).astype(npdt)
    gref = O.vm_backward(sc, cam, ref, G, dtype=npdt)
    grads = cpp_binding.backward(*ts, cam.width, cam.height, cam.tan_fovx, cam.tan_fovy, sc.sh_degree,
                                 torch.tensor(G, device=dev), cache)
    for name, g in zip(GRAD_NAMES, grads):
        e = grad_err(g.cpu().numpy().reshape(gref[name].shape), gref[name])
        assert e <= GRAD_TOL, (name, e)
    r = ref["i_ranges"].reshape(-1, 2)
    return int((r[:, 1] - r[:, 0]).max())


@pytest.mark.parametrize("n,dtype", [(500, torch.float32), (1023, torch.float32), (1100, torch.float32),
                                     (500, torch.float64), (530, torch.float64)])
def test_more_usable_entries_than_a_ray_keeps(cuda, n, dtype):
    """A small dense cluster: the rays through its middle can use every Gaussian."""
    sc = S.make_scene(n, seed=n, extent=0.02, scale_range=(0.04, 0.05))
    sc.weights = np.random.default_rng(n).uniform(0.01, 0.05, size=n).astype(np.float32)
    check(sc, S.make_camera(33, 17, eye=(0.1, 0.05, -0.9)), cuda, dtype)


def test_tile_list_longer_than_16_bit_offsets(cuda):
    """Every Gaussian lies on one of a few tiles; one in a hundred has the mass to be used."""
    n = 68_000
    sc = S.make_scene(n, seed=9, extent=0.4, scale_range=(0.01, 0.02))
    rng = np.random.default_rng(9)
    sc.weights = np.where(rng.random(n) < 0.01, rng.uniform(0.2, 0.9, size=n), 1e-4).astype(np.float32)
    assert check(sc, S.make_camera(16, 16), cuda, torch.float32) > 65_536


@pytest.mark.parametrize("n,extent,scales,eye,size", [
    (3000, 1.0, (0.0005, 0.5), (0.0, 0.0, -3.0), (40, 24)),  # needles and plates, 1000 to 1
    (2000, 0.5, (0.005, 0.05), (0.1, 0.0, -0.3), (24, 24)),  # from inside the cloud
    (3000, 30.0, (0.2, 2.0), (3.0, 1.0, -60.0), (32, 32)),  # far away
    (20000, 1.0, (0.005, 0.05), (0.0, 0.0, -2.5), (16, 16)),  # many candidates per ray, most turned away
])
def test_entries_turned_away_are_not_usable(cuda, n, extent, scales, eye, size):
    """The approximate test on a Gaussian's record turns away no entry that the
    exact one would use: the march fills as many bins as the oracle."""
    sc = S.make_scene(n, seed=n, extent=extent, scale_range=scales)
    cam = S.make_camera(*size, eye=eye)
    with O.decision_audit() as audit:
        O.vm_forward(sc, cam)
    counter = torch.zeros(1, dtype=torch.int64, device=cuda)
    cache, ts = run_vm(sc, cam, cuda, torch.float32)
    cpp_binding.forward(*ts, cam.width, cam.height, cam.tan_fovx, cam.tan_fovy, sc.sh_degree, work_counter=counter)
    assert int(counter.item()) == audit["fills"] > 0
    check(sc, cam, cuda, torch.float32)
