"""The work that users of this package have it do, as cases that can be timed.

Every case goes through the package's public entry points: the splat renderer
(`splat.splat_forward`, `splat.render` under autograd), the volume marcher
(`vol_marcher.apply`, `cpp_binding.forward` / `backward`), the volume
rasteriser, batches of views under CUDA graphs, and the continuous server.

Scenes are drawn as everywhere in this repository: centres uniform in a cube,
per-axis scales log-uniform in [0.005, 0.05], random rotations, opacity
sigmoid(N(0, 1)), colours uniform in [0, 1] as the SH constant term (and small
higher terms where the SH degree asks for them).  Cameras look at the origin
from a distance of 2.5 to 4.

`listed()` names the cases, `draw(rng)` gives more of the same ranges,
`prepare` / `run` execute one, `work` says what a pass cannot do without and
`exact` evaluates the splat cases in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from differentiable_gaussian_mixture_renderer_b200 import cpp_binding, splat, vol_marcher, vol_raster
from differentiable_gaussian_mixture_renderer_b200 import scene as S
from differentiable_gaussian_mixture_renderer_b200.batch import BatchRenderer
from differentiable_gaussian_mixture_renderer_b200.serving import GaussianScene, NativeServer, ServeRequest

SCALES = (0.005, 0.05)
# the view sizes of the batch and serving workloads
SIZES = ((256, 256), (800, 600), (1920, 1080), (512, 512), (1280, 720))


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a preview or a small test frame: host work, launches and their gaps count
        dict(name="splat_forward_10k_256", kind="splat", n=10_000, width=256, height=256, extent=1.0, sh=0, train=False),
        # a viewer's frame: one large scene at full HD, forward only, sized from its own pair count
        dict(name="splat_forward_1m_1080p", kind="splat", n=1_000_000, width=1920, height=1080, extent=1.0, sh=0, train=False),
        # a training step of the splat renderer: forward and all five gradients
        dict(name="splat_train_200k_1024", kind="splat", n=200_000, width=1024, height=1024, extent=2.0, sh=0, train=True),
        # the same with view-dependent colour (16 SH coefficients) and a frame that is no multiple of a tile
        dict(name="splat_train_sh3_300k_801x603", kind="splat", n=300_000, width=801, height=603, extent=1.0, sh=3, train=True),
        # the largest training step
        dict(name="splat_train_1m_1080p", kind="splat", n=1_000_000, width=1920, height=1080, extent=1.0, sh=0, train=True),
        # a small marched frame without gradients
        dict(name="march_forward_10k_256", kind="march", n=10_000, width=256, height=256, extent=1.0, sh=0, train=False, f64=False, recompute=False),
        # a training step of the volume marcher through its autograd op
        dict(name="march_train_100k_512", kind="march", n=100_000, width=512, height=512, extent=1.0, sh=0, train=True, f64=False, recompute=False),
        # a gradient check: float64, through the binding, whose backward recomputes the samples; odd frame
        dict(name="march_binding_f64_4k_97x65", kind="march", n=4_000, width=97, height=65, extent=1.0, sh=1, train=True, f64=True, recompute=True),
        # a frame of the volume rasteriser
        dict(name="raster_100k_512", kind="raster", n=100_000, width=512, height=512, extent=1.0, sh=0),
        # a training step over several scenes and cameras of mixed sizes, one captured sequence
        dict(name="batch_splat_train_12_views", kind="batch_splat", scenes=3, n_min=50_000, n_max=1_500_000, views=12),
        # many small marched views in one captured sequence (patches of a training step)
        dict(name="batch_march_train_16x64", kind="batch_march", n=100_000, width=64, height=64, views=16),
        # a render server: requests on several resident scenes, a quarter of them with gradients
        dict(name="serve_mixed_16_requests", kind="serve", scenes=4, n_min=100_000, n_max=1_500_000, requests=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["splat", "splat", "splat", "march", "march", "raster", "batch_splat", "batch_march", "serve"])
    if kind == "splat":
        return dict(kind=kind, n=_log(rng, 2_000, 1_000_000), width=_log(rng, 128, 1920), height=_log(rng, 128, 1080),
                    extent=rng.choice([1.0, 2.0]), sh=rng.choice([0, 0, 1, 2, 3]), train=rng.random() < 0.5)
    if kind == "march":
        if rng.random() < 0.25:
            return dict(kind=kind, n=_log(rng, 1_000, 5_000), width=_log(rng, 32, 120), height=_log(rng, 32, 120), extent=1.0,
                        sh=rng.choice([0, 1]), train=True, f64=True, recompute=True)
        train = rng.random() < 0.6
        return dict(kind=kind, n=_log(rng, 2_000, 90_000), width=_log(rng, 64, 500), height=_log(rng, 64, 500), extent=1.0,
                    sh=rng.choice([0, 0, 3]), train=train, f64=False, recompute=train and rng.random() < 0.4)
    if kind == "raster":
        return dict(kind=kind, n=_log(rng, 2_000, 100_000), width=_log(rng, 64, 512), height=_log(rng, 64, 512), extent=1.0, sh=rng.choice([0, 2]))
    if kind == "batch_splat":
        return dict(kind=kind, scenes=rng.randint(1, 3), n_min=_log(rng, 5_000, 50_000), n_max=_log(rng, 50_000, 1_500_000), views=rng.randint(2, 12))
    if kind == "batch_march":
        return dict(kind=kind, n=_log(rng, 5_000, 100_000), width=_log(rng, 24, 64), height=_log(rng, 24, 64), views=rng.randint(2, 16))
    return dict(kind=kind, scenes=rng.randint(1, 4), n_min=_log(rng, 10_000, 100_000), n_max=_log(rng, 100_000, 1_500_000), requests=rng.randint(4, 16))


# ----------------------------------------------------------------- the inputs
def _scene(n, extent, sh, seed, dtype=torch.float32):
    """(shs, opacity, means, scales, rotations) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    o = dict(device="cuda", dtype=torch.float32, generator=g)
    means = (torch.rand((n, 3), **o) * 2 - 1) * extent
    lo, hi = math.log(SCALES[0]), math.log(SCALES[1])
    scales = torch.exp(torch.rand((n, 3), **o) * (hi - lo) + lo)
    q = torch.randn((n, 4), **o)
    q = q / q.norm(dim=1, keepdim=True)
    opacity = torch.sigmoid(torch.randn((n, 1), **o))
    shs = torch.randn((n, (sh + 1) ** 2, 3), **o) * 0.1
    shs[:, 0] = (torch.rand((n, 3), **o) - 0.5) / S.SH_C0
    return tuple(t.to(dtype).contiguous() for t in (shs, opacity, means, scales, q))


def _image_grad(width, height, seed, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(seed + 7919)
    return torch.randn((3, height, width), device="cuda", dtype=torch.float32, generator=g).to(dtype)


def _cuda_camera(cam, dtype=torch.float32):
    """The camera as a training script holds it: tensors on the GPU."""
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")  # noqa: E731
    return t(cam.view), t(cam.proj), t(cam.campos), torch.zeros(3, dtype=dtype, device="cuda")


def _counts(case):
    """Gaussian counts of a multi-scene case, log-spaced."""
    k = case["scenes"]
    if k == 1:
        return [case["n_max"]]
    r = math.log(case["n_max"] / case["n_min"]) / (k - 1)
    return [int(round(case["n_min"] * math.exp(r * i))) for i in range(k)]


def _requests(case):
    """(scene, width, height, with gradients) of each view of a multi-scene case."""
    got = []
    for i in range(case["views"] if "views" in case else case["requests"]):
        w, h = SIZES[i % 3] if case["kind"] == "batch_splat" else SIZES[i % 5]
        got.append((i % case["scenes"], w, h, case["kind"] == "batch_splat" or i % 4 == 1))
    return got


def _multi(case, seed):
    """The scenes, cameras and image gradients of a multi-scene case."""
    scenes = [_scene(n, 1.0, 0, 1000 * seed + 31 * k + 1) for k, n in enumerate(_counts(case))]
    views = []
    for i, (k, w, h, grad) in enumerate(_requests(case)):
        cam = S.random_cameras(1, w, h, seed=1000 * seed + i)[0]
        views.append((k, cam, _image_grad(w, h, 1000 * seed + i) if grad else None))
    return scenes, views


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("splat", "march", "raster"):
        dtype = torch.float64 if case.get("f64") else torch.float32
        tensors = _scene(case["n"], case["extent"], case["sh"], seed, dtype)
        cam = S.random_cameras(1, case["width"], case["height"], seed=seed)[0]
        st = dict(case=case, tensors=tensors, cam=cam, cuda_cam=_cuda_camera(cam, dtype))
        if case.get("train"):
            st["tensors"] = tuple(t.requires_grad_(not case.get("recompute")) for t in tensors)
            st["grad"] = _image_grad(case["width"], case["height"], seed, dtype)
        return st
    if kind == "batch_march":
        tensors = _scene(case["n"], 1.0, 0, seed)
        scenes = {0: GaussianScene(*tensors[:1], tensors[1].reshape(-1), *tensors[2:], 0)}
        views = [(0, c) for c in S.random_cameras(case["views"], case["width"], case["height"], seed=seed)]
        grads = [_image_grad(case["width"], case["height"], 1000 * seed + i) for i in range(case["views"])]
        return dict(case=case, **_captured(scenes, views, grads, "march"))
    if kind == "batch_splat":
        tensors, views = _multi(case, seed)
        scenes = {k: GaussianScene(t[0], t[1].reshape(-1), *t[2:], 0) for k, t in enumerate(tensors)}
        return dict(case=case, **_captured(scenes, [(k, c) for k, c, _ in views], [g for _, _, g in views], "splat"))
    tensors, views = _multi(case, seed)
    scenes = {k: GaussianScene(t[0], t[1].reshape(-1), *t[2:], 0) for k, t in enumerate(tensors)}
    return dict(case=case, server=NativeServer(scenes, n_slots=4, max_batch=8), views=views)


def _captured(scenes, views, grads, kind):
    renderer = BatchRenderer(scenes, kind=kind)
    plan = renderer.plan(views, backward=True)
    for to, g in zip(plan.grad_framebuffers, grads):
        to.copy_(g)
    return dict(renderer=renderer, plan=renderer.capture(plan, backward=True))


# -------------------------------------------------------------------- a pass
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("splat", "march", "raster"):
        t, cam = state["tensors"], state["cam"]
        args = (*t, *state["cuda_cam"], cam.width, cam.height, cam.tan_fovx, cam.tan_fovy, case["sh"])
        if kind == "raster":
            return vol_raster.forward(*args)
        if not case["train"]:
            if kind == "splat":
                return splat.splat_forward(*args)[0]
            with torch.no_grad():
                return vol_marcher.apply(*args)
        if case.get("recompute"):
            cache = cpp_binding.forward(*args)
            return [cache[0], *cpp_binding.backward(*args, state["grad"], cache)]
        image = (splat.render if kind == "splat" else vol_marcher.apply)(*args)
        return [image.detach(), *torch.autograd.grad(image, t, state["grad"])]
    if kind in ("batch_splat", "batch_march"):
        plan = state["plan"]
        state["renderer"].replay(plan)
        return [*plan.framebuffers, *(list(plan.grads[k]) for k in plan.scene_ids)]
    server = state["server"]
    reqs = [server.submit(ServeRequest(k, cam, backward=grad is not None, grad_image=grad)) for k, cam, grad in state["views"]]
    server.drain()
    server.completed.clear()
    return [[r.image, *(r.grads or ())] for r in reqs]


# ------------------------------------------------- what a pass cannot do without
def _splat_work(n, sh, width, height, train, extent=1.0):
    """Inputs read once and outputs written once; per Gaussian the projection
    (and its adjoint), per covered pixel the blend step (and its adjoint)."""
    k = (sh + 1) ** 2
    params = 4.0 * n * (3 * k + 11)
    image = 12.0 * width * height
    # mean squared screen-space scale at a distance of 3.2, and the area of the ellipse where alpha >= 1/255
    s2 = (SCALES[1] ** 2 - SCALES[0] ** 2) / (2 * math.log(SCALES[1] / SCALES[0])) * (height / (2 * math.tan(math.pi / 6)) / 3.2) ** 2 + 0.3
    covered = min(n * 2 * math.pi * s2 * 4.0 / extent ** 2, 150.0 * width * height)
    flops = 400.0 * n + 35.0 * covered
    if train:
        return dict(bytes=2 * params + 2 * image, flops=flops + 900.0 * n + 60.0 * covered)
    return dict(bytes=params + image, flops=flops)


def _march_work(n, sh, width, height, train, extent=1.0, size=4.0):
    """As above; per Gaussian that a ray meets, 128 borders of a CDF (35
    operations each) and their adjoint."""
    w = _splat_work(n, sh, width, height, train, extent)
    s2 = (SCALES[1] ** 2 - SCALES[0] ** 2) / (2 * math.log(SCALES[1] / SCALES[0])) * (height / (2 * math.tan(math.pi / 6)) / 3.2) ** 2 + 0.3
    met = min(n * 2 * math.pi * s2 * 2.0 / extent ** 2, 60.0 * width * height)
    return dict(bytes=w["bytes"] * size / 4, flops=1300.0 * n + met * 128 * 35.0 * (2.5 if train else 1.0))


def work(case):
    kind = case["kind"]
    if kind == "splat":
        return _splat_work(case["n"], case["sh"], case["width"], case["height"], case["train"], case["extent"])
    if kind == "march":
        return _march_work(case["n"], case["sh"], case["width"], case["height"], case["train"], case["extent"], 8.0 if case["f64"] else 4.0)
    if kind == "raster":  # 32 bins, each fitted and integrated in 256 steps of about 10 operations
        w = _march_work(case["n"], case["sh"], case["width"], case["height"], False, case["extent"])
        return dict(bytes=w["bytes"], flops=w["flops"] / 4 + 32 * 256 * 10.0 * case["width"] * case["height"])
    total = dict(bytes=0.0, flops=0.0)
    if kind == "batch_march":
        parts = [_march_work(case["n"], 0, case["width"], case["height"], True) for _ in range(case["views"])]
        total["bytes"] -= 2 * 4.0 * 14 * case["n"] * (case["views"] - 1)  # the scene is read, and its gradient written, once
    else:
        counts = _counts(case)
        parts = [_splat_work(counts[k], 0, w, h, grad) for k, w, h, grad in _requests(case)]
    for p in parts:
        total = {m: total[m] + p[m] for m in total}
    return total


# --------------------------------------------------- the splat cases in 64 bits
def _project(t, cam, sh_degree):
    """Screen-space splats of a scene, differentiable: EWA projection with the
    1.3 tan(fov) clamp, a 0.3 pixel filter and the weight that keeps a
    Gaussian's mass over its two larger axes; SH colour."""
    shs, opacity, mu, s, q = t
    view, proj = (torch.as_tensor(np.asarray(m, dtype=np.float64), device=mu.device) for m in (cam.view, cam.proj))
    campos = torch.as_tensor(np.asarray(cam.campos, dtype=np.float64), device=mu.device)
    h = torch.cat([mu, torch.ones_like(mu[:, :1])], 1)
    tu, pp = h @ view, h @ proj
    fx, fy = cam.width / (2 * cam.tan_fovx), cam.height / (2 * cam.tan_fovy)
    z = tu[:, 2]
    x = torch.maximum(torch.minimum(tu[:, 0], 1.3 * cam.tan_fovx * z), -1.3 * cam.tan_fovx * z)
    y = torch.maximum(torch.minimum(tu[:, 1], 1.3 * cam.tan_fovy * z), -1.3 * cam.tan_fovy * z)
    length, zero = torch.sqrt(x * x + y * y + z * z), torch.zeros_like(z)
    J = torch.stack([torch.stack([fx / z, zero, -fx * x / z ** 2], 1), torch.stack([zero, fy / z, -fy * y / z ** 2], 1),
                     torch.stack([x, y, z], 1) / length[:, None]], 1)
    w_, i, j, k = q.unbind(1)
    R = torch.stack([1 - 2 * (j * j + k * k), 2 * (i * j - w_ * k), 2 * (i * k + w_ * j),
                     2 * (i * j + w_ * k), 1 - 2 * (i * i + k * k), 2 * (j * k - w_ * i),
                     2 * (i * k - w_ * j), 2 * (j * k + w_ * i), 1 - 2 * (i * i + j * j)], 1).reshape(-1, 3, 3)
    M = J[:, :2] @ view[:3, :3].T @ (R * s[:, None, :])
    cov = M @ M.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    two = torch.sort(s, dim=1).values
    weight = opacity.reshape(-1) * torch.linalg.det(J) * (2 * math.pi * two[:, 1] * two[:, 2]) / (2 * math.pi * torch.sqrt(det))
    d = pp[:, 3] + 1e-7
    xy = torch.stack([((pp[:, 0] / d + 1) * cam.width - 1) / 2, ((pp[:, 1] / d + 1) * cam.height - 1) / 2], 1)
    away = mu - campos
    depth = away.norm(dim=1)
    rgb = _colour(shs, away / depth[:, None], sh_degree)
    return xy, torch.stack([c / det, -b / det, a / det], 1), weight, rgb, depth.detach(), tu[:, 2].detach(), a.detach(), c.detach()


def _colour(sh, direction, degree):
    x, y, z = (direction[:, i, None] for i in range(3))
    r = 0.28209479177387814 * sh[:, 0]
    if degree > 0:
        r = r + 0.4886025119029199 * (-y * sh[:, 1] + z * sh[:, 2] - x * sh[:, 3])
    if degree > 1:
        r = r + 1.0925484305920792 * (x * y * sh[:, 4] - y * z * sh[:, 5] - x * z * sh[:, 7])
        r = r + 0.31539156525252005 * (2 * z * z - x * x - y * y) * sh[:, 6] + 0.5462742152960396 * (x * x - y * y) * sh[:, 8]
    if degree > 2:
        r = r - 0.5900435899266435 * (y * (3 * x * x - y * y) * sh[:, 9] + x * (x * x - 3 * y * y) * sh[:, 15])
        r = r + 2.890611442640554 * x * y * z * sh[:, 10] + 1.445305721320277 * z * (x * x - y * y) * sh[:, 14]
        r = r - 0.4570457994644658 * (4 * z * z - x * x - y * y) * (y * sh[:, 11] + x * sh[:, 13])
        r = r + 0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y) * sh[:, 12]
    return torch.clamp(r + 0.5, min=0.0)


def _exact_splat(tensors, cam, sh_degree, grad=None):
    """[image] or [image, five gradients] of one frame in 64 bits: every
    16x16 tile's splats front to back, in groups of tiles with lists of like
    length."""
    leaves = [t.detach().double().requires_grad_(grad is not None) for t in tensors]
    W, H = cam.width, cam.height
    xy, conic, weight, rgb, depth, vz, va, vc = _project(leaves, cam, sh_degree)
    flat = [t.detach().requires_grad_(grad is not None) for t in (xy, conic, weight, rgb)]
    gx, gy = (W + 15) // 16, (H + 15) // 16
    with torch.no_grad():
        ex, ey = torch.ceil(3 * torch.sqrt(va)), torch.ceil(3 * torch.sqrt(vc))
        cut = lambda v, g: torch.trunc(v / 16).clamp(0, g).long()  # noqa: E731
        x0, x1 = cut(xy[:, 0] - ex, gx), cut(xy[:, 0] + ex + 15, gx)
        y0, y1 = cut(xy[:, 1] - ey, gy), cut(xy[:, 1] + ey + 15, gy)
        count = torch.where(vz < 0.2, 0, (x1 - x0) * (y1 - y0))
        order = torch.sort(depth, stable=True).indices
        order = order[count[order] > 0]
        who = torch.repeat_interleave(order, count[order])
        first = torch.cumsum(count[order], 0) - count[order]
        at = torch.arange(who.numel(), device=who.device) - torch.repeat_interleave(first, count[order])
        wide = (x1 - x0)[who]
        tile = (y0[who] + at // wide) * gx + x0[who] + at % wide
        tile, by = torch.sort(tile, stable=True)
        who = who[by]
        length = torch.bincount(tile, minlength=gx * gy)
        start = torch.cumsum(length, 0) - length
        todo = torch.sort(length, descending=True).indices.tolist()
        sizes = length.tolist()
    image = torch.zeros((3, gy * 16, gx * 16), dtype=torch.float64, device=who.device)
    lane = torch.arange(16, device=who.device, dtype=torch.float64)
    i = 0
    while i < len(todo) and sizes[todo[i]] > 0:
        n = sizes[todo[i]]
        k = max(1, min(len(todo) - i, 24_000_000 // (n * 256)))
        ids = torch.tensor([t for t in todo[i:i + k] if sizes[t] > 0], device=who.device)
        i += k
        pos = torch.arange(n, device=who.device)
        have = pos[None, :] < length[ids][:, None]
        g = who[(start[ids][:, None] + pos).clamp(max=who.numel() - 1)]
        px = ((ids % gx) * 16)[:, None, None, None] + lane[None, None, None, :]
        py = ((ids // gx) * 16)[:, None, None, None] + lane[None, None, :, None]
        dx, dy = px - flat[0][g][..., 0, None, None], py - flat[0][g][..., 1, None, None]
        Q = flat[1][g][..., None, None]
        alpha = flat[2][g][..., None, None] * torch.exp(-0.5 * (Q[:, :, 0] * dx * dx + 2 * Q[:, :, 1] * dx * dy + Q[:, :, 2] * dy * dy))
        alpha = torch.clamp(alpha, max=0.99)
        alpha = torch.where((alpha >= 1 / 255) & have[..., None, None], alpha, 0.0)
        after = torch.cumprod(1 - alpha.detach(), 1)
        alpha = torch.where(after >= 1e-4, alpha, 0.0)
        after = torch.cumprod(1 - alpha, 1)
        before = torch.cat([torch.ones_like(after[:, :1]), after[:, :-1]], 1)
        tiles = torch.einsum("tnij,tnc->tcij", alpha * before, flat[3][g])
        for to, t in zip(ids.tolist(), tiles.detach()):
            image[:, to // gx * 16:to // gx * 16 + 16, to % gx * 16:to % gx * 16 + 16] = t
        if grad is not None:
            back = torch.nn.functional.pad(grad.double(), (0, gx * 16 - W, 0, gy * 16 - H))
            back = back.reshape(3, gy, 16, gx, 16).permute(1, 3, 0, 2, 4).reshape(-1, 3, 16, 16)[ids]
            tiles.backward(back)
        del alpha, after, before, tiles, dx, dy, Q
    image = image[:, :H, :W].contiguous()
    if grad is None:
        return [image]
    mine = [(v, f.grad) for v, f in zip((xy, conic, weight, rgb), flat) if f.grad is not None]
    # splats on no tile take no part: their projection may be undefined
    seen = torch.zeros_like(count, dtype=torch.bool)
    seen[who] = True
    torch.autograd.backward([v for v, _ in mine], [g for _, g in mine])
    out = []
    for t in leaves:
        keep = seen.reshape(-1, *[1] * (t.dim() - 1))
        out.append(torch.where(keep, t.grad if t.grad is not None else torch.zeros_like(t), 0.0))
    return [image, *out]


def exact(case, seed):
    """The splat cases as the definition says, in 64 bits.  The marched and
    the rasterised images have no such value here: where a ray is sampled
    follows from a chain of insertions into a bounded set, entry by entry, and
    plain torch or numpy walks that chain for minutes."""
    kind = case["kind"]
    if kind == "splat":
        t = _scene(case["n"], case["extent"], case["sh"], seed)
        cam = S.random_cameras(1, case["width"], case["height"], seed=seed)[0]
        got = _exact_splat(t, cam, case["sh"], _image_grad(case["width"], case["height"], seed) if case["train"] else None)
        return got if case["train"] else got[0]
    if kind not in ("batch_splat", "serve"):
        return None
    scenes, views = _multi(case, seed)
    got = [_exact_splat(scenes[k], cam, 0, g) for k, cam, g in views]
    if kind == "serve":
        return [[r[0]] + ([r[1], r[2].reshape(-1), *r[3:]] if len(r) > 1 else []) for r in got]
    ids = list(dict.fromkeys(k for k, _, _ in views))
    sums = [[sum(r[1 + m] for r, (k, _, _) in zip(got, views) if k == s) for m in range(5)] for s in ids]
    return [*(r[0] for r in got), *([g[0], g[1].reshape(-1), *g[2:]] for g in sums)]
