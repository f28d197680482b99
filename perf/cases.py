"""The work that a user of the rasterizer has it do, as measurable cases: `listed()` names some, `draw()` gives more of the
same ranges, `prepare()` makes what a program has in hand before the call, `run()` is one pass through the public entry
points, `work()` is what a pass cannot do without and `tolerance()` how far two correct results may be apart.

A case is a dict of plain values. Its "kind":

  step        one training step of the rasterizer, forward and backward, by one of two public interfaces: "rasterizer" =
              adop_b200.raster.PointRasterizer with outputs that are kept from step to step, "operator" = the libTorch
              autograd operator torch.ops.adop.blend_point_cloud[_environment], which allocates its outputs
  view        one frame of a viewer: the forward pass alone, nothing recorded for a backward pass, descriptors unchanged
  tonemap     photometric tonemapper forward and backward through torch.ops.adop.tonemap (autograd)
  preprocess  what a scene's point cloud goes through once when it is loaded: Morton reorder, block shuffle, neighbour
              radius, radius sort inside the blocks, and the rows moved along
"""
import math

import numpy as np
import torch

from adop_b200 import build, capi, preprocess, synth
from adop_b200.raster import PointRasterizer, Scene

DEV = "cuda:0"


def _raster_case(name, kind, **kw):
    c = dict(name=name, kind=kind, api="rasterizer", scene="surfaces", order="morton", model="pinhole", points=0, views=1, w=0, h=0,
             layers=4, channels=4, env=True, crops=False, dropout=0.0, radius=False, normals=False, index=False)
    c.update(kw)
    return c


def listed():
    return [
        # A preview window over a small cloud: launches and host work are all there is.
        _raster_case("view_small", "view", points=60_000, w=320, h=180),
        # A unit-test sized training step through autograd (drop-out as in training): latency again, both directions.
        _raster_case("step_small", "step", api="operator", scene="frustum", points=20_011, w=135, h=77, layers=3, env=False, dropout=0.25),
        # One view of an object-sized cloud, the benchmark's smallest configuration: 2^20 points, 512 x 512, identity pose.
        _raster_case("step_object", "step", scene="frustum", points=1 << 20, w=512, h=512, env=False),
        # The reference's training loop as it ships: a batch of random 512 x 512 crops, drop-out, radius rule and normal test
        # on, cloud in the order its preprocessing leaves (blocks of 256 points, shuffled, sorted by radius), shared texels.
        _raster_case("step_crops", "step", api="operator", order="shuffled", points=3_000_000, views=4, w=512, h=512, layers=5, crops=True,
                     dropout=0.25, radius=True, normals=True, index=True),
        # Fisheye rig with uneven sizes: omnidirectional model, eight channels, drop-out.
        _raster_case("step_fisheye", "step", scene="box", model="ocam", points=2_345_677, views=2, w=1237, h=731, layers=5, channels=8,
                     env=False, dropout=0.25),
        # The benchmark's training scene: 10 M points, 16 views of 1080p, environment map, every gradient.
        _raster_case("step_training", "step", points=10_000_000, views=16, w=1920, h=1080),
        # One GPU's share of the view-sharded configuration: 30 M points, 8 views of 1080p.
        _raster_case("step_large_scene", "step", points=30_000_000, views=8, w=1920, h=1080),
        # The HDR configuration: 50 M points, 4 views of 4K, six layers, eight channels.
        _raster_case("step_hdr", "step", points=50_000_000, views=4, w=3840, h=2160, layers=6, channels=8),
        # The real-time viewer: 100 M points through the omnidirectional model, one 1080p frame.
        _raster_case("view_large", "view", scene="box", model="ocam", points=100_000_000, w=1920, h=1080, env=False),
        # The tonemapper on a batch of training crops with a short response curve, and on the HDR configuration's 4K frames.
        dict(name="tonemap_crops", kind="tonemap", batch=4, w=509, h=383, bins=25, leak=0.01),
        dict(name="tonemap_hdr", kind="tonemap", batch=4, w=3840, h=2160, bins=256, leak=0.01),
        # Loading the benchmark's training scene for the first time.
        dict(name="preprocess_scene", kind="preprocess", points=10_000_000, normals=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["step", "step", "step", "step", "view", "view", "tonemap", "preprocess"])
    if what == "tonemap":
        pixels = _log_int(rng, 40_000, 8_000_000)
        w = max(64, min(3840, int(math.sqrt(pixels * rng.uniform(1.0, 1.9)))))
        return dict(kind="tonemap", batch=rng.randint(1, 4), w=w, h=max(48, pixels // w), bins=rng.choice([2, 25, 64, 256, 300, 1024]),
                    leak=rng.choice([0.0, 0.01]))
    if what == "preprocess":
        return dict(kind="preprocess", points=_log_int(rng, 50_000, 10_000_000), normals=rng.random() < 0.5)
    points = _log_int(rng, 20_000, 40_000_000)
    w = _log_int(rng, 128, 1920)
    h = max(64, min(1080, int(w * rng.uniform(0.5, 1.0))))
    model = "ocam" if rng.random() < 0.25 else "pinhole"
    c = _raster_case(None, what, points=points, w=w, h=h, layers=rng.randint(3, 5), channels=rng.choice([3, 4, 4, 4, 8, 16]), model=model,
                     scene="box" if model == "ocam" else rng.choice(["surfaces", "surfaces", "frustum"]),
                     order=rng.choice(["morton", "shuffled"]), env=model == "pinhole" and rng.random() < 0.7)
    del c["name"]
    if what == "step":
        c["api"] = rng.choice(["rasterizer", "operator"])
        budget = 100_000_000 // (1 if c["channels"] <= 4 else c["channels"] // 4)
        c["views"] = max(1, min(_log_int(rng, 1, 16), budget // points))
        c["crops"] = model == "pinhole" and c["scene"] == "surfaces" and rng.random() < 0.5
        c["dropout"] = rng.choice([0.0, 0.25])
        c["radius"], c["normals"], c["index"] = rng.random() < 0.4, rng.random() < 0.4, rng.random() < 0.3
    return c


# ---- inputs -------------------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _surface_cloud(n, seed, g):
    """Points (and normals) on 64 random spheres and square patches, radii U[0.2,2], centres U[-1.5,1.5]^3, N(0,0.005) noise."""
    rng = np.random.default_rng(seed)
    m = 64
    sphere = rng.integers(0, 2, m) == 0
    radius = rng.uniform(0.2, 2.0, m)
    centre = rng.uniform(-1.5, 1.5, (m, 3))
    a = rng.normal(size=(m, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(m, 3)))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    area = np.where(sphere, 4 * math.pi * radius ** 2, 4 * radius ** 2)
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float32, device=DEV)
    first = np.concatenate([[0], np.round(np.cumsum(area) / area.sum() * n).astype(np.int64)])
    xyz = torch.empty((n, 3), device=DEV)
    normal = torch.empty((n, 3), device=DEV)
    for k in range(m):
        lo, hi = int(first[k]), int(first[k + 1])
        if hi <= lo:
            continue
        c, r = t(centre[k]), float(radius[k])
        if sphere[k]:
            d = torch.nn.functional.normalize(torch.randn((hi - lo, 3), device=DEV, generator=g), dim=1)
            xyz[lo:hi] = c + r * d
            normal[lo:hi] = d
        else:
            uv = (torch.rand((hi - lo, 2), device=DEV, generator=g) * 2 - 1) * r
            xyz[lo:hi] = c + uv[:, :1] * t(a[k]) + uv[:, 1:] * t(b[k])
            normal[lo:hi] = t(np.cross(a[k], b[k]))
    xyz += 0.005 * torch.randn((n, 3), device=DEV, generator=g)
    return xyz, normal, math.sqrt(area.sum() / n)


def _cloud(kind, n, seed, g):
    """(xyz [n,3], unit normals [n,3], typical distance between neighbours)."""
    if kind == "surfaces":
        return _surface_cloud(n, seed, g)
    xyz = torch.empty((n, 3), device=DEV)
    if kind == "frustum":   # in front of a camera at the origin that looks along +z
        xyz[:, :2] = torch.randn((n, 2), device=DEV, generator=g)
        xyz[:, 2] = torch.rand(n, device=DEV, generator=g) * 4 + 2
        spacing = (50.0 / n) ** (1 / 3)
    else:                   # a flat box around the camera
        xyz.copy_((torch.rand((n, 3), device=DEV, generator=g) * 2 - 1) * torch.tensor([10.0, 10.0, 2.5], device=DEV))
        spacing = (2000.0 / n) ** (1 / 3)
    normal = torch.nn.functional.normalize(torch.randn((n, 3), device=DEV, generator=g), dim=1) if n <= 40_000_000 else None
    return xyz, normal, spacing


def _pack_normals(v):
    q = torch.round((v + 1) * (0.5 * 1023)).to(torch.int32)
    return (q[:, 0] | (q[:, 1] << 10) | (q[:, 2] << 20)).contiguous()


def _rows(t, order):
    return preprocess.permute_rows(t, order)


def _prepare_raster(c, seed):
    g = _generator(seed)
    rng = np.random.default_rng(seed + 1)
    n, B, w, h, L, C = c["points"], c["views"], c["w"], c["h"], c["layers"], c["channels"]
    xyz, nrm, spacing = _cloud(c["scene"], n, seed, g)
    pos = torch.empty((n, 4), device=DEV)
    pos[:, :3] = xyz
    del xyz
    pos[:, 3] = 0.01
    if c["radius"]:
        pos[:, 3] = spacing * torch.rsqrt(1.0 - torch.rand(n, device=DEV, generator=g))
    normal = _pack_normals(nrm) if c["normals"] else None
    del nrm
    # what the scene's preprocessing does once, when it is loaded
    orders = [preprocess.morton_order(pos)]
    if c["order"] == "shuffled":
        orders.append(preprocess.block_shuffle_order(n, DEV, 256, seed=seed & 0xffff))
    for o in orders:
        pos, normal = _rows(pos, o), _rows(normal, o) if normal is not None else None
    if c["order"] == "shuffled":
        o = preprocess.sort_blocks_by_radius_order(pos)
        pos, normal = _rows(pos, o), _rows(normal, o) if normal is not None else None
    index, texels = None, n
    if c["index"]:          # neighbours share a descriptor, as after the cloud was densified
        texels = (n + 1) // 2
        index = torch.arange(n, device=DEV, dtype=torch.int32) // 2
    texture = torch.randn((C, texels), device=DEV, generator=g) * 0.1 + 0.5
    background = torch.rand(C, device=DEV, generator=g)
    params = capi.default_render_params()
    params.dropout, params.dropout_seed = c["dropout"], seed & 0xffffff
    params.drop_out_points_by_radius, params.check_normal = int(c["radius"]), int(c["normals"])
    params.output_background_mask = int(c["env"])
    params.composite_environment_map = int(c["env"])
    env = torch.rand((C, 512, 1024) if w * h < 4_000_000 else (C, 1024, 2048), device=DEV, generator=g) if c["env"] else None
    if c["model"] == "ocam":
        s = w / 1920.0
        coef, theta_max = synth.ocam_world2cam_poly((-300.0 * s, 0.0, 5e-4 / s, -1e-7 / (s * s)), rho_max=1150.0 * s)
        intr = np.concatenate([[1, 0, 0, w / 2, h / 2], coef])[None]
        params.dist_cutoff = float(math.tan(theta_max) * 0.98)
    else:
        full_w, full_h = (1920, 1080) if c["crops"] else (w, h)
        f = 1400.0 * full_w / 1920.0 if c["scene"] == "surfaces" else 500.0 * w / 512.0
        intr = np.array([[f, f, full_w / 2, full_h / 2, 0, -0.1, 0.02, 0, 0, 0, 0, 0, 0]])
    if c["scene"] == "surfaces":
        turn = rng.uniform(0, 2 * math.pi)
        poses = np.stack([synth.look_at_pose((4 * math.cos(turn + 2 * math.pi * i / B), 0.3 * math.sin(turn + 4 * math.pi * i / B),
                                              4 * math.sin(turn + 2 * math.pi * i / B))) for i in range(B)])
    else:                   # cameras at the origin that look along +z, each turned and moved a little
        poses = np.stack([synth.look_at_pose(rng.normal(0, 0.02, 3) * (i > 0), rng.normal(0, 0.1, 3) * (i > 0) + (0, 0, 4), (0, -1, 0.01))
                          for i in range(B)])
    views = []
    for i in range(B):
        v = dict(w=w, h=h, image_index=i, camera_index=0,
                 camera_model=capi.CAMERA_OCAM if c["model"] == "ocam" else capi.CAMERA_PINHOLE_DISTORTION)
        if c["crops"]:      # a window of the full image, zoomed
            z = math.exp(rng.uniform(math.log(0.6), math.log(1.4)))
            v["crop"] = (z, z, -rng.uniform(0, max(0.0, 1920 * z - w)), -rng.uniform(0, max(0.0, 1080 * z - h)), 0.0)
        views.append(v)
    t = lambda a, d=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=DEV)
    scene = Scene(pos, texture, background, t(poses, torch.float64), t(intr), normal=normal, index=index, env_map=env)
    state = dict(kind=c["kind"], scene=scene, views=capi.make_views(views), params=params, layers=L, want_env=env is not None)
    if c["kind"] == "step":
        state["grads"] = [torch.randn((B, C, hh, ww), device=DEV, generator=g) for ww, hh in capi.layer_sizes(w, h, L)]
    if c["api"] == "rasterizer":
        state["rasterizer"] = PointRasterizer(DEV)
        state["fwd"] = state["bwd"] = None
        return state
    torch.ops.load_library(build.TORCH_OP_LIB)
    info = torch.classes.adop.RenderInfo()
    info.set_scene(scene.poses, normal, index, None)
    info.set_views(torch.tensor([[v["w"], v["h"], v["image_index"], 0, v["camera_model"]] for v in views]),
                   torch.tensor([list(v.get("crop", (1.0, 1.0, 0.0, 0.0, 0.0))) for v in views], dtype=torch.float32))
    info.set_num_layers(L)
    for name, _ in type(params)._fields_:
        info.set_param(name, float(getattr(params, name)))
    leaves = dict(texture=texture, background=background, points=pos,
                  tangents=torch.zeros((B, 6), dtype=torch.float64, device=DEV), intrinsics=scene.intrinsics)
    if env is not None:
        leaves["env_map"] = env
    for v in leaves.values():
        v.requires_grad_(True)
    state.update(rasterizer=None, info=info, leaves=leaves)
    return state


def _tonemap_inputs(c, seed):
    g = _generator(seed)
    B, w, h = c["batch"], c["w"], c["h"]
    # exposed frames: smooth shading with grain, darks near 0 and highlights that clip
    shade = torch.nn.functional.interpolate(torch.rand((B, 3, 9, 16), device=DEV, generator=g), size=(h, w), mode="bicubic", align_corners=True)
    x = shade * 1.15 + 0.02 * torch.randn((B, 3, h, w), device=DEV, generator=g)
    ev = torch.rand((B, 1, 1, 1), device=DEV, generator=g) * 4 - 2
    x = (x * torch.exp2(ev)).contiguous()
    wb = 1 + 0.05 * torch.randn((B, 3, 1, 1), device=DEV, generator=g)
    wb[:, 1] = 1.0
    response = (torch.linspace(0, 1, c["bins"], device=DEV) ** (1 / 2.2)).repeat(1, 3, 1).contiguous()
    leaves = dict(x=x, exposures=ev, white_balance=wb, vignette=torch.tensor([0.1, -0.05, 0.01], device=DEV),
                  centre=torch.zeros((1, 2, 1, 1), device=DEV), response=response)
    return leaves, torch.randn((B, 3, h, w), device=DEV, generator=g)


def _prepare_tonemap(c, seed):
    torch.ops.load_library(build.TORCH_OP_LIB)
    leaves, grad = _tonemap_inputs(c, seed)
    for v in leaves.values():
        v.requires_grad_(True)
    return dict(kind="tonemap", leaves=leaves, frames=torch.arange(c["batch"], device=DEV, dtype=torch.int32), size=(c["w"], c["h"]),
                leak=c["leak"], grad=grad)


def _prepare_preprocess(c, seed):
    g = _generator(seed)
    n = c["points"]
    xyz, nrm, _ = _surface_cloud(n, seed, g)
    pos = torch.zeros((n, 4), device=DEV)
    pos[:, :3] = xyz
    shuffle = torch.randperm(n, device=DEV, generator=g)  # a file's order follows the images it was triangulated from, not space
    return dict(kind="preprocess", position=pos[shuffle].contiguous(), seed=seed & 0xffff,
                normal=_pack_normals(nrm[shuffle]) if c["normals"] else None)


def prepare(case, seed):
    if case["kind"] == "tonemap":
        return _prepare_tonemap(case, seed)
    if case["kind"] == "preprocess":
        return _prepare_preprocess(case, seed)
    return _prepare_raster(case, seed)


# ---- one pass -----------------------------------------------------------------------------------------------------------
def _run_rasterizer(s):
    r, scene, step = s["rasterizer"], s["scene"], s["kind"] == "step"
    # a viewer's descriptors do not change between frames; a training step's do
    fwd = s["fwd"] = r.forward(scene, s["views"], s["params"], s["layers"], out=s["fwd"], record_visible=step, refresh_descriptors=step)
    out = dict(color=fwd.colors, mask=fwd.masks, depth=fwd.depths, weight=fwd.weights)
    if step:
        out["grad"] = s["bwd"] = r.backward(scene, s["params"], fwd, s["grads"], want_env=s["want_env"], out=s["bwd"])
    return out


def _run_operator(s):
    a, L = s["leaves"], s["layers"]
    args = (a["texture"], a["background"], a["points"], a["tangents"], a["intrinsics"])
    if "env_map" in a:
        images = torch.ops.adop.blend_point_cloud_environment(*args, a["env_map"], s["info"])
    else:
        images = torch.ops.adop.blend_point_cloud(*args, s["info"])
    grads = torch.autograd.grad(images[:L], list(a.values()), s["grads"])
    return dict(images=[t.detach() for t in images], grad=list(grads))


def _run_tonemap(s):
    a = s["leaves"]
    out = torch.ops.adop.tonemap(a["x"], s["frames"], None, a["exposures"], a["white_balance"], a["vignette"], a["centre"], a["response"],
                                 s["size"][0], s["size"][1], s["leak"])
    grads = torch.autograd.grad(out, list(a.values()), s["grad"])
    return dict(image=out.detach(), grad=list(grads))


def _run_preprocess(s):
    pos, normal = s["position"], s["normal"]
    n = pos.shape[0]
    morton = preprocess.morton_order(pos)
    pos = preprocess.permute_rows(pos, morton)
    shuffle = preprocess.block_shuffle_order(n, DEV, 256, seed=s["seed"])
    pos = preprocess.permute_rows(pos, shuffle)
    pos[:, 3] = preprocess.radius_sample(preprocess.knn_distance(pos, k=4), seed=s["seed"])
    by_radius = preprocess.sort_blocks_by_radius_order(pos)
    pos = preprocess.permute_rows(pos, by_radius)
    if normal is not None:
        for order in (morton, shuffle, by_radius):
            normal = preprocess.permute_rows(normal, order)
    return dict(morton=morton, shuffle=shuffle, by_radius=by_radius, position=pos, normal=normal)


def run(state):
    if state["kind"] == "tonemap":
        return _run_tonemap(state)
    if state["kind"] == "preprocess":
        return _run_preprocess(state)
    return _run_rasterizer(state) if state["rasterizer"] is not None else _run_operator(state)


# ---- what a pass cannot do without, and how far results may be apart ---------------------------------------------------
def work(case):
    if case["kind"] == "tonemap":
        px = case["batch"] * case["w"] * case["h"]
        return dict(bytes=48 * px, flops=200 * px)   # image in and out, upstream gradient in, gradient out
    if case["kind"] == "preprocess":
        n = case["points"]
        return dict(bytes=n * (16 + 16 + 3 * 4 + (8 if case["normals"] else 0)), flops=100 * n)
    c = case
    n, B, C = c["points"], c["views"], c["channels"]
    texels = (n + 1) // 2 if c["index"] else n
    pixels = B * sum(ww * hh for ww, hh in capi.layer_sizes(c["w"], c["h"], c["layers"]))
    env = (4 * C * (512 * 1024 if c["w"] * c["h"] < 4_000_000 else 1024 * 2048)) if c["env"] else 0
    cloud = n * (16 + (4 if c["normals"] else 0) + (4 if c["index"] else 0)) + 4 * C * texels
    images = pixels * (4 * C + 8 + (4 if c["env"] else 0))   # colour, depth, weight, mask
    total = cloud + images + env
    if c["kind"] == "step":
        # upstream gradients in; descriptor, point and environment-map gradients out
        total += 4 * C * pixels + 4 * C * texels + 16 * n + env
    return dict(bytes=total, flops=n * B * 50 + (pixels * C * 60 if c["kind"] == "step" else pixels * C * 10))


def tolerance(case):
    if case["kind"] == "preprocess":
        return "exact"   # permutations and exact float32 distances
    # float32 sums of up to millions of terms in the GPU's order. Seen between the same pass twice, and between the pass over
    # the recorded lists and the one over all points: rel up to 2.4e-6 (intrinsics gradient), max up to 1.3e-5 (environment map).
    return {"rel": 1e-5, "max": 6e-5}


# ---- the same numbers in 64 bits ----------------------------------------------------------------------------------------
def _exact_tonemap(c, seed):
    leaves, grad = _tonemap_inputs(c, seed)
    a = {k: v.double().requires_grad_(True) for k, v in leaves.items()}
    B, w, h, K, leak = c["batch"], c["w"], c["h"], c["bins"], c["leak"]
    yy, xx = torch.meshgrid(torch.linspace(-1, 1, h, device=DEV, dtype=torch.float64), torch.linspace(-1, 1, w, device=DEV, dtype=torch.float64),
                            indexing="ij")
    images, grads = [], None
    for b in range(B):      # an image at a time: eight bytes a value, and several values a pixel
        du, dv = (xx - a["centre"][0, 0, 0, 0]) * (w / h), yy - a["centre"][0, 1, 0, 0]
        r2 = du * du + dv * dv
        vig = a["vignette"]
        v = (1 + r2 * (vig[0] + r2 * (vig[1] + r2 * vig[2]))) * (a["white_balance"][b] * (a["x"][b] * torch.exp2(-a["exposures"][b])))
        z = v.detach()
        t = z.clamp(0, 1) * (K - 1)
        i0 = t.floor().long()
        fr = t - i0
        row = torch.arange(3, device=DEV).view(3, 1, 1) * K
        lo, hi = row + i0, row + (i0 + 1).clamp(max=K - 1)
        curve = a["response"].detach().reshape(-1)
        out = curve[lo] * (1 - fr) + curve[hi] * fr
        slope = (curve[hi] - curve[lo]) * (K - 1) * ((z > 0) & (z < 1))
        if leak > 0:
            knee = z.abs() + 1e-4
            out = out + torch.where(z < 0, leak * z, torch.where(z > 1, leak - leak * knee ** -0.5, 0.0))
            slope = slope + torch.where(z < 0, leak, torch.where(z > 1, 0.5 * leak * knee ** -1.5, 0.0))
        images.append(out)
        up = grad[b].double()
        part = list(torch.autograd.grad(v, [a[k] for k in ("x", "exposures", "white_balance", "vignette", "centre")], up * slope))
        bins = torch.bincount(lo.reshape(-1), (up * (1 - fr)).reshape(-1), 3 * K) + torch.bincount(hi.reshape(-1), (up * fr).reshape(-1), 3 * K)
        part.append(bins.view_as(a["response"]))
        grads = part if grads is None else [p + q for p, q in zip(grads, part)]
    return dict(image=torch.stack(images), grad=grads)


def exact(case, seed):
    """The tonemapper in 64 bits. The rasterizer has no such value: which pixel a point rounds to and whether it passes the depth
    test are decided on float32 numbers, and 64-bit ones decide some of them differently, which moves whole splats. The
    preprocessing's results are permutations and float32 distances that are compared bit by bit."""
    return _exact_tonemap(case, seed) if case["kind"] == "tonemap" else None
