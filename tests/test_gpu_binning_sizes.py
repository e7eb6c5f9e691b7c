"""The binning's dispatch at the sizes where it changes: one-, two- and
three-launch scans over the Gaussians, super-tile plans from one sort pass and
from two, tile scans of one and several steps and beyond one block.  Checked
against their definition: offsets are the running sum of the tile counts; every
tile's list is its Gaussians in (depth bits, index) order, each where its
rectangle covers the tile."""
import numpy as np
import pytest
import torch

from differentiable_gaussian_mixture_renderer_b200 import scene as S
from test_gpu_parity import run_splat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h,extent", [
    (16_384, 256, 256, 1.0), (16_385, 256, 256, 1.0),  # scans: one block, two launches
    (2048 * 2048, 64, 64, 60.0), (2048 * 2048 + 1, 64, 64, 60.0),  # two launches, three
    (5_000, 2048, 2048, 1.5), (5_000, 2176, 2176, 1.5),  # 256 super-tiles: one sort pass; 289: two
    (5_000, 2048, 1024, 1.5), (5_000, 2064, 1024, 1.5),  # 8192 tiles: one step of the tile scan; 8256: two
    (5_000, 3000, 3000, 1.5),  # 35,344 tiles: past the one-block scan
    (1, 16, 16, 0.1),
])
def test_binning_is_its_definition(cuda, n, w, h, extent):
    sc = S.make_scene(n, seed=1, extent=extent)
    cam = S.make_camera(w, h)
    _, frame, _ = run_splat(sc, cam, cuda)
    v = {k: t.cpu().numpy() for k, t in frame.views().items()}
    gx, gy = (w + 15) // 16, (h + 15) // 16
    counts = v["tiles_touched"].astype(np.int64)
    np.testing.assert_array_equal(v["point_offsets"], np.cumsum(counts))
    P = int(counts.sum())
    assert [int(x) for x in frame.stats.tolist()][:2] == [P, 0] and P > 0
    seen = np.flatnonzero(counts)
    xy, e = v["points_xy_image"][seen], v["rects"][seen].astype(np.float32)
    cut = lambda a, g: np.clip(np.trunc(a / np.float32(16)).astype(np.int64), 0, g)  # noqa: E731
    x0, x1 = cut(xy[:, 0] - e[:, 0], gx), cut(xy[:, 0] + e[:, 0] + np.float32(16) - np.float32(1), gx)
    y0 = cut(xy[:, 1] - e[:, 1], gy)
    reps = counts[seen]
    who = np.repeat(seen, reps)
    k = np.arange(P) - np.repeat(np.cumsum(reps) - reps, reps)
    wide = np.repeat(x1 - x0, reps)
    tile = (np.repeat(y0, reps) + k // wide) * gx + np.repeat(x0, reps) + k % wide
    order = np.lexsort((who, v["depths"].view(np.uint32)[who], tile))
    np.testing.assert_array_equal(v["point_list"][:P], who[order])
    np.testing.assert_array_equal(v["point_list_tiles"][:P], tile[order])
    per_tile = np.bincount(tile, minlength=gx * gy)
    end = np.cumsum(per_tile)
    want = np.where(per_tile[:, None] > 0, np.stack([end - per_tile, end], 1), 0)
    np.testing.assert_array_equal(v["i_ranges"], want)
