"""A splat frame's workspaces stay the size they are, so that every frame that
fits the static 64 MiB of dgmr_splat_forward_noalloc keeps fitting."""
import pytest

from differentiable_gaussian_mixture_renderer_b200 import _native


@pytest.mark.parametrize("n,w,h,frame", [(100_000, 512, 512, 21_098_496), (200_000, 256, 256, 38_000_384), (1, 16, 16, 8_960)])
def test_splat_workspaces_have_not_grown(n, w, h, frame):
    lib = _native.load()
    assert lib.dgmr_splat_frame_workspace_size(n, w, h) <= frame
    assert lib.dgmr_splat_pair_workspace_size(n, 5_000_000) <= 83_752_704
