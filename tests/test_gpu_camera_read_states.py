"""Reading a camera on the device inside a graph capture: refused, without a mark
on the capture or on the calls that follow."""
import threading

import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import _native as N, scene as S
from test_gpu_camera_read import struct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["relaxed", "thread_local", "global"])
def test_a_read_inside_a_capture_is_only_refused(cuda, mode):
    cam = S.random_cameras(1, 64, 48, seed=4)[0]
    host = [torch.as_tensor(np.asarray(a), dtype=torch.float32) for a in (cam.view, cam.proj, cam.campos, (0.1, 0.2, 0.3))]
    dev = [t.to(cuda) for t in host]
    want = struct(*host)
    x = torch.zeros(8, device=cuda)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        graph.capture_begin(capture_error_mode=mode)
        x.add_(1.0)
        with pytest.raises(N.DgmrError):
            struct(*dev)
        x.add_(1.0)
        graph.capture_end()
    assert struct(*dev) == want
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8


def test_a_thread_that_has_read_may_end_beside_a_capture(cuda):
    """What the thread keeps for its reads is freed when it ends; that is no part of
    another thread's capture."""
    cam = S.random_cameras(1, 64, 48, seed=4)[0]
    host = [torch.as_tensor(np.asarray(a), dtype=torch.float32) for a in (cam.view, cam.proj, cam.campos, (0.1, 0.2, 0.3))]
    dev = [t.to(cuda) for t in host]
    got, read, end = [], threading.Event(), threading.Event()

    def work():
        got.append(struct(*dev))
        read.set()
        end.wait(30)

    t = threading.Thread(target=work)
    t.start()
    assert read.wait(30)
    x = torch.zeros(8, device=cuda)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        x.add_(1.0)
        end.set()
        t.join()
        x.add_(1.0)
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8 and got == [struct(*host)]
