"""A camera given as device tensors is read in one go, one given any other way
array by array: the same struct."""
import ctypes as C

import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import _native as N, scene as S

pytestmark = pytest.mark.gpu


def struct(*arrays):
    return bytes(N.make_camera(*arrays, 64, 48, 0.7, 0.5))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
def test_device_and_host_cameras_agree(cuda, dtype):
    cam = S.random_cameras(1, 64, 48, seed=4)[0]
    host = [torch.as_tensor(np.asarray(a), dtype=dtype) for a in (cam.view, cam.proj, cam.campos, (0.1, 0.2, 0.3))]
    want = struct(*host)
    dev = [t.to(cuda) for t in host]
    assert struct(*dev) == want
    # transposed storage, more values than are read, a mixture, a tensor that requires grad
    assert struct(dev[0].T.contiguous().T, dev[1], dev[2], dev[3]) == want
    assert struct(dev[0], dev[1], torch.cat([dev[2], dev[2]]), dev[3]) == want
    assert struct(dev[0], host[1], dev[2], [float(v) for v in host[3]]) == want
    assert struct(dev[0], dev[1], dev[2].clone().requires_grad_(True), dev[3]) == want
    assert struct(dev[0], dev[1].double(), dev[2], dev[3]) == want
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        late = [torch.zeros_like(t) for t in dev]
        for to, t in zip(late, dev):
            to.copy_(t)
        assert struct(*late) == want


def test_short_arrays_are_refused(cuda):
    t = lambda n: torch.ones(n, device=cuda)  # noqa: E731
    with pytest.raises(IndexError):
        N.make_camera(t(16), t(12), t(3), t(3), 8, 8, 1.0, 1.0)


def test_null_arrays_are_refused(cuda):
    cam = N.Camera()
    assert N.lib().dgmr_camera_read(None, None, None, None, 0, C.byref(cam), None) == N.DGMR_ERR_BAD_ARG
