"""The measured cases of the voxel ray-traversal library, through its public entry points.

listed() and draw() give cases (dicts of plain values), prepare() what a user's
program holds before a call, run() one pass through the entry points, work()
what a pass cannot do without, exact() the floating-point outputs in 64 bits.

The kinds, and what each stands for:

  rays       vt_trace_rays on a ray list: line-of-sight tests, picking, a lidar sweep
  frame      vt_render: one camera's frame into device memory
  host       vt_render_host: the same into pinned host memory (a host without CUDA code)
  batch      vt_batch_launch: many small scenes, several cameras each
  shade      vt_shade_forward_views + vt_shade_backward_views: one iteration of an
             inverse-rendering fit (zeroed gradients, images, loss, gradients)
  edit       a game loop's two frames of editing: place a voxel, draw, remove it, draw
  generate   a level made on the device and its first frame (empty-space distances
             are built by that frame)
  reference  vt_render_reference: the frame of the original engine's format, bit for bit
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "unnamed-voxel-tracer_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import vt  # noqa: E402

_RAYS = {"primary": vt.RAYS_PRIMARY, "shadow": vt.RAYS_PRIMARY | vt.RAYS_SHADOW,
         "bounce": vt.RAYS_PRIMARY | vt.RAYS_SHADOW | vt.RAYS_BOUNCE}
_SHADE = {"none": vt.SHADE_NONE, "reference": vt.SHADE_REFERENCE, "lambert": vt.SHADE_LAMBERT}
_SIZES = ((320, 240), (640, 480), (1280, 720), (1920, 1080))


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # A few hundred line-of-sight rays of a game tick: one launch's latency.
        {"name": "rays_500", "kind": "rays", "x": 128, "y": 128, "z": 128, "trees": 0, "caves": False, "rays": 500},
        # A lidar-like sweep: a million unrelated rays in a terrain world (not a multiple of a block).
        {"name": "rays_1m", "kind": "rays", "x": 512, "y": 256, "z": 512, "trees": 200, "caves": False,
         "rays": 1000003},
        # A preview frame of a small world, primary rays only: launch and tail bound.
        {"name": "frame_360p", "kind": "frame", "x": 128, "y": 128, "z": 128, "trees": 0, "caves": False,
         "width": 640, "height": 360, "rays": "primary", "shade": "reference", "entities": 0},
        # The ordinary game frame: 1080p, shadows.
        {"name": "frame_1080p", "kind": "frame", "x": 512, "y": 256, "z": 512, "trees": 200, "caves": False,
         "width": 1920, "height": 1080, "rays": "shadow", "shade": "reference", "entities": 0},
        # Ragged everything: world sides off the brick and chunk grid, an odd image, Lambert shading, entity
        # occluders in the shadow pass, one bounce ray per hit.
        {"name": "frame_odd", "kind": "frame", "x": 301, "y": 107, "z": 173, "trees": 40, "caves": True,
         "width": 1021, "height": 577, "rays": "bounce", "shade": "lambert", "entities": 12},
        # The largest frame: 4K over a 1 GiB cave world, shadow and bounce rays.
        {"name": "frame_4k_bounce", "kind": "frame", "x": 2048, "y": 256, "z": 2048, "trees": 3200, "caves": True,
         "width": 3840, "height": 2160, "rays": "bounce", "shade": "reference", "entities": 0},
        # The game frame read by a host program: records into pinned memory.
        {"name": "host_1080p", "kind": "host", "x": 512, "y": 256, "z": 512, "trees": 200, "caves": False,
         "width": 1920, "height": 1080, "rays": "shadow", "shade": "reference", "entities": 0},
        # Data-set rendering: 16 cube scenes of 32 to 448 voxels, 1-4 cameras each, 320x240 to 1080p.
        {"name": "batch_16", "kind": "batch", "scenes": 16, "edge_lo": 32, "edge_hi": 448, "rays": "shadow"},
        # One iteration of fitting a palette, per-voxel albedo and sun to 16 views.
        {"name": "shade_16x512", "kind": "shade", "x": 256, "y": 256, "z": 256, "trees": 50, "caves": False,
         "views": 16, "width": 512, "height": 512},
        # Building in the game: place and remove a voxel, a small frame after each.
        {"name": "edit_512", "kind": "edit", "x": 512, "y": 256, "z": 512, "trees": 200, "caves": False,
         "width": 640, "height": 360},
        # Level load: a cave world generated on the device, then its first frame.
        {"name": "generate_512", "kind": "generate", "x": 512, "y": 256, "z": 512, "trees": 200, "caves": True,
         "width": 640, "height": 360},
        # The original engine's world and frame.
        {"name": "reference_1080p", "kind": "reference", "width": 1920, "height": 1080},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, sizes spread over the ranges of the listed ones."""
    kind = rng.choice(["rays", "frame", "frame", "host", "batch", "shade", "edit", "generate", "reference"])
    if kind == "batch":
        lo = _log(rng, 32, 96)
        return {"kind": kind, "scenes": _log(rng, 3, 16), "edge_lo": lo, "edge_hi": _log(rng, 2 * lo, 448),
                "rays": rng.choice(["primary", "shadow"])}
    if kind == "reference":
        w = _log(rng, 320, 1920)
        return {"kind": kind, "width": w, "height": max(180, int(w * rng.uniform(0.5, 0.6)))}
    case = {"kind": kind, "x": _log(rng, 64, 512), "y": _log(rng, 48, 256), "z": _log(rng, 64, 512),
            "trees": rng.randrange(0, 200), "caves": rng.random() < 0.5}
    if kind == "rays":
        case["rays"] = _log(rng, 100, 1000003)
    elif kind == "shade":
        for a in "xyz":
            case[a] = min(case[a], 256)
        case.update(views=rng.randrange(1, 17), width=_log(rng, 128, 512), height=_log(rng, 128, 512))
    elif kind in ("frame", "host"):
        w = _log(rng, 320, 3840 if kind == "frame" else 1920)
        case.update(width=w, height=max(180, int(w * rng.uniform(0.45, 0.6))),
                    rays=rng.choice(["primary", "shadow", "bounce"] if kind == "frame" else ["primary", "shadow"]),
                    shade=rng.choice(["reference", "lambert", "none"]), entities=rng.choice([0, 0, 5, 12]))
    else:
        case.update(width=_log(rng, 320, 640), height=_log(rng, 180, 360))
    return case


# ------------------------------------------------------------------- the state
class _Tensor(vt.DeviceBuffer):
    """A torch tensor as the device buffer the host binding takes."""

    def __init__(self, ctx, tensor):
        self.ctx, self.tensor = ctx, tensor
        self.ptr, self.nbytes = tensor.data_ptr(), tensor.numel() * tensor.element_size()

    def free(self):
        self.tensor = self.ptr = None


class _View:
    """Library memory as an array that keeps its owner alive."""

    def __init__(self, owner, interface):
        self.owner = owner
        self.__dict__[interface[0]] = interface[1]


class _Held:
    """A context and the objects made in it, released together in order."""

    def __init__(self):
        self.ctx = vt.Context(0)
        self.objects = []

    def add(self, obj):
        self.objects.append(obj)
        return obj

    def device_view(self, ptr, count, typestr, dtype):
        v = _View(self, ("__cuda_array_interface__", {"data": (int(ptr), False), "shape": (count,),
                                                      "typestr": typestr, "version": 3}))
        return torch.as_tensor(v, device="cuda").view(dtype)

    def __del__(self):
        for obj in reversed(self.objects):
            (obj.close if hasattr(obj, "close") else obj.free)()
        self.ctx.close()


def _records(count):
    return torch.zeros((count, 4), dtype=torch.int32, device="cuda")


def _desc(case, seed):
    """Terrain whose height suits the world's: the default generator at y / 128, at most full size."""
    return vt.gen_desc((case["x"], case["y"], case["z"]), scale=min(1.0, case["y"] / 128.0), seed=seed,
                       trees=case["trees"], caves=case["caves"])


def _world(held, desc):
    world = held.add(vt.World(held.ctx, tuple(desc.dims)))
    world.generate(desc)
    return world


def _params(case, seed):
    return vt.default_params(rays=_RAYS[case["rays"]], shade=_SHADE[case.get("shade", "reference")], seed=seed,
                             max_steps=512, shadow_max_steps=512, bounce_max_steps=256, sun_dir=vt.gen_sun(seed))


def _entities(rng, case, n):
    lo = rng.uniform(0.0, 1.0, (n, 3)) * (case["x"], case["y"], case["z"])
    return np.concatenate([lo, lo + rng.uniform(1.0, 6.0, (n, 3))], axis=1)


def _looking_down(desc, seed, width, height):
    """A camera over the seeded column whose centre ray meets the ground."""
    at = vt.gen_camera(desc, seed, width, height)
    return vt.Camera(pos=list(at.pos)[:3], yaw=0.7 * seed, pitch=-0.6, fov=math.radians(70.0), width=width,
                     height=height).as_uniform_data()


def _reference_world(held, rng, seed):
    chunks, bricks = vt.procgen_reference(512, seed=seed)
    bm = held.add(vt.Brickmap(held.ctx))
    bm.upload(chunks, bricks)
    types = int((bricks & 0xFFFFFFF).max()) + 1
    for slot in range(min(types, 32)):
        keep = rng.random((8, 8, 8)) < rng.uniform(0.4, 1.0)
        texels = rng.integers(0, 1 << 24, (8, 8, 8)).astype(np.uint32) | np.uint32(0xFF000000)
        bm.set_model(slot, np.where(keep, texels, 0))
    x, z = (int(v) for v in rng.integers(64, 448, 2))
    column = chunks.reshape(64, 64, 64)[z >> 3, :, x >> 3]
    voxels = bricks.reshape(-1, 8, 8, 8)
    top = max((8 * b + int(np.flatnonzero(voxels[c - 1, z & 7, :, x & 7])[-1])
               for b, c in enumerate(column) if c and voxels[c - 1, z & 7, :, x & 7].any()), default=0)
    return bm, (x + 0.5, top + 11.5, z + 0.5)


def prepare(case, seed):
    kind = case["kind"]
    held = _Held()
    ctx = held.ctx
    rng = np.random.default_rng(seed)
    state = {"case": case, "held": held}
    if kind == "batch":
        n = case["scenes"]
        jobs, k = [], 0
        for s in range(n):
            edge = int(round(case["edge_lo"] * (case["edge_hi"] / case["edge_lo"]) ** (s / (n - 1))))
            desc = vt.gen_desc((edge, edge, edge), scale=edge / 128.0, seed=1000 * seed + s)
            world = _world(held, desc)
            for c in range(1 + (5 * s) % 4):
                w, h = _SIZES[k % 4]
                jobs.append((world, vt.gen_camera(desc, seed + c, w, h)))
                k += 1
        out = _records(sum(cam.width * cam.height for _, cam in jobs))
        at, full = 0, []
        for world, cam in jobs:
            full.append((world, cam, _Tensor(ctx, out[at:at + cam.width * cam.height])))
            at += cam.width * cam.height
        state["out"] = out
        state["batch"] = held.add(vt.Batch(ctx, full, _params(case, seed)))
        return state
    if kind == "reference":
        state["world"], pos = _reference_world(held, rng, seed)
        state["cam"] = vt.Camera(pos=pos, yaw=float(rng.uniform(0.0, 6.28)), pitch=float(rng.uniform(-0.5, 0.0)),
                                 fov=math.radians(70.0), width=case["width"], height=case["height"]).as_uniform_data()
        state["out"] = torch.zeros((case["width"] * case["height"], 8), dtype=torch.int32, device="cuda")
        return state

    desc = _desc(case, seed)
    world = state["world"] = _world(held, desc)
    if kind == "rays":
        n = case["rays"]
        size = np.array([case["x"], case["y"], case["z"]])
        o = rng.uniform(0.0, 1.0, (n, 3)) * size
        o[:, 1] = (0.3 + 0.7 * o[:, 1] / size[1]) * size[1]
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        state["o"] = torch.from_numpy(o.astype(np.float32)).cuda()
        state["d"] = torch.from_numpy(d.astype(np.float32)).cuda()
        state["out"] = _records(n)
        return state

    w, h = case["width"], case["height"]
    if kind == "shade":
        cams = state["cams"] = [vt.gen_camera(desc, 100 * seed + v, w, h) for v in range(case["views"])]
        hits, images = [_records(w * h) for _ in cams], torch.zeros((len(cams), h, w, 3), device="cuda")
        state["hits"], state["images"], state["targets"] = hits, images, torch.zeros_like(images)
        state["d_hits"] = [_Tensor(ctx, t) for t in hits]
        state["d_images"] = [_Tensor(ctx, t) for t in images]
        state["d_targets"] = [_Tensor(ctx, t) for t in state["targets"]]
        for cam, d_hits in zip(cams, state["d_hits"]):
            vt.render(ctx, world, cam, vt.default_params(rays=vt.RAYS_PRIMARY, shade=vt.SHADE_NONE), d_hits)
        cells = case["x"] * case["y"] * case["z"]
        albedo = rng.uniform(0.5, 1.5, cells).astype(np.float32)
        hidden = rng.uniform(0.05, 0.95, (256, 3)).astype(np.float32)
        sh = state["shading"] = held.add(vt.Shading(ctx, world, hidden, albedo, vt.gen_sun(seed + 200)))
        sh.forward_views(cams, state["d_hits"], state["d_targets"])
        ctx.sync()
        palette, sun = rng.uniform(0.05, 0.95, (256, 3)).astype(np.float32), vt.gen_sun(seed + 100)
        sh.set_params(palette, albedo, sun)
        state["fit"] = (palette, albedo, sun)
        grads = state["grads"] = {"loss": torch.zeros(1, device="cuda"), "palette": torch.zeros((256, 3), device="cuda"),
                                  "albedo": torch.zeros(cells, device="cuda"), "sun": torch.zeros(3, device="cuda")}
        for name, attr in (("loss", "d_loss"), ("palette", "d_gpal"), ("albedo", "d_galb"), ("sun", "d_gsun")):
            getattr(sh, attr).free()
            setattr(sh, attr, _Tensor(ctx, grads[name]))
        return state
    if kind == "generate":
        info = world.info()
        state["desc"] = desc
        state["materials"] = held.device_view(info.d_materials, info.material_bytes, "|u1", torch.uint8)
        state["mask"] = held.device_view(info.d_mask, info.mask_bytes // 8, "<i8", torch.int64)
    if kind == "edit":
        state["cam"] = _looking_down(desc, seed, w, h)
        state["picks"] = _records(2)
        state["d_picks"] = [_Tensor(ctx, t) for t in state["picks"]]
    else:
        state["cam"] = vt.gen_camera(desc, seed, w, h)
    if case.get("entities"):
        world.set_entities(_entities(rng, case, case["entities"]))
    state["params"] = _params({"rays": "shadow", **case}, seed)
    if kind == "host":
        pinned = held.add(vt.PinnedBuffer(ctx, w * h, vt.HIT_DTYPE))
        state["out"] = np.asarray(_View(held, ("__array_interface__", {
            "data": (pinned.ptr, False), "shape": (w * h,), "typestr": "|V16", "version": 3}))).view(vt.HIT_DTYPE)
    else:
        frames = state["frames"] = [_records(w * h) for _ in range(2 if kind == "edit" else 1)]
        state["d_frames"] = [_Tensor(ctx, t) for t in frames]
    return state


# -------------------------------------------------------------------- one pass
def run(state):
    case, ctx = state["case"], state["held"].ctx
    kind = case["kind"]
    if kind == "batch":
        state["batch"].launch()
        return state["out"]
    world = state["world"]
    if kind == "rays":
        ctx.check(ctx.lib.vt_trace_rays(ctx.handle, world.handle, state["o"].data_ptr(), state["d"].data_ptr(),
                                        case["rays"], 512, state["out"].data_ptr(), None))
        return state["out"]
    if kind == "reference":
        ctx.check(ctx.lib.vt_render_reference(ctx.handle, world.handle, state["cam"], state["out"].data_ptr(), None))
        return state["out"]
    if kind == "shade":
        sh = state["shading"]
        sh.zero_grad_async()
        sh.forward_views(state["cams"], state["d_hits"], state["d_images"])
        sh.backward_views(state["cams"], state["d_hits"], state["d_targets"])
        return {"images": state["images"], **state["grads"]}
    cam, params = state["cam"], state["params"]
    if kind == "host":
        return vt.render_host(ctx, world, cam, params, state["out"]).view(np.int32)
    if kind == "edit":
        for mode, d_pick, d_frame in zip((7, 0), state["d_picks"], state["d_frames"]):
            world.edit(cam, 256, mode, d_pick)
            vt.render(ctx, world, cam, params, d_frame)
        return {"picks": state["picks"], "frames": state["frames"]}
    if kind == "generate":
        world.generate(state["desc"])
        vt.render(ctx, world, cam, params, state["d_frames"][0])
        return {"materials": state["materials"], "mask": state["mask"], "frame": state["frames"][0]}
    vt.render(ctx, world, cam, params, state["d_frames"][0])
    return state["frames"][0]


def work(case):
    """Bytes: each record written once, and per ray the 8-byte brick word and the material byte it ends at.
    Flops: a ray's set-up and one cell crossing (about 40), shading and generation as noted."""
    kind = case["kind"]
    rays_per_pixel = {"primary": 1, "shadow": 2, "bounce": 3}
    if kind == "batch":
        n = case["scenes"]
        jobs = sum(1 + (5 * s) % 4 for s in range(n))
        px = sum(_SIZES[k % 4][0] * _SIZES[k % 4][1] for k in range(jobs))
        r = rays_per_pixel[case["rays"]]
        return {"bytes": px * (16 + 9 * r), "flops": px * 40 * r}
    if kind == "rays":
        return {"bytes": case["rays"] * (24 + 9 + 16), "flops": case["rays"] * 40}
    px = case["width"] * case["height"]
    if kind == "reference":
        return {"bytes": px * (32 + 2 * 12), "flops": px * 80}
    cells = case["x"] * case["y"] * case["z"]
    if kind == "shade":
        px *= case["views"]
        # records read twice, images written, targets read, a shadow ray each way; gradients cleared and written
        return {"bytes": px * (2 * 16 + 12 + 12 + 2 * 8) + 2 * 4 * cells, "flops": px * 140}
    if kind == "edit":
        return {"bytes": 2 * px * (16 + 18), "flops": 2 * px * 80}
    if kind == "generate":
        # materials, occupancy bits and the eight direction fields of the distances written once; cave noise of the
        # lower half of the cells: two octaves of 7 interpolations (3 operations each)
        return {"bytes": cells * (1 + 1 / 8 + 1 / 8) + px * (16 + 18),
                "flops": (cells / 2 * 42 if case["caves"] else 0) + px * 80}
    r = rays_per_pixel[case["rays"]]
    return {"bytes": px * (16 + 9 * r), "flops": px * 40 * r}


# ------------------------------------------------------------- 64-bit results
def _blocked(solid, o, d, max_steps):
    """Whether the rays o + t d meet a solid cell before leaving the grid: unit steps in 64 bits, at most
    max_steps cells tested, the origin's own cell first."""
    size = torch.tensor(solid.shape[::-1], device=o.device)
    hit = torch.zeros(o.shape[0], dtype=torch.bool, device=o.device)
    ids = torch.arange(o.shape[0], device=o.device)
    step = torch.where(d > 0, 1, -1)
    cell = torch.floor(o).long()
    inv = 1.0 / d
    t = ((cell + (step > 0)).double() - o) * inv
    for _ in range(max_steps):
        inside = ((cell >= 0) & (cell < size)).all(1)
        c = torch.minimum(cell.clamp(min=0), size - 1)
        now = inside & solid[c[:, 2], c[:, 1], c[:, 0]]
        hit[ids[now]] = True
        go = inside & ~now
        if not bool(go.any()):
            break
        ids, cell, t, step, inv = ids[go], cell[go], t[go], step[go], inv[go]
        axis = torch.argmin(t, 1, keepdim=True)
        cell = cell.scatter_add(1, axis, step.gather(1, axis))
        t = t.scatter_add(1, axis, inv.gather(1, axis).abs())
    return hit


def exact(case, seed):
    """The shading case in 64 bits from the same inputs (hit records, targets, parameters). The other kinds return
    whole numbers and bytes (records, voxels), which have no such value."""
    if case["kind"] != "shade":
        return None
    s = prepare(case, seed)
    palette, albedo, sun = (torch.from_numpy(np.asarray(v, np.float64)).cuda() for v in s["fit"])
    solid = torch.from_numpy(s["world"].download_dense() != 0).cuda()
    ambient, diffuse = (float(np.float32(v)) for v in (0.2, 0.8))
    length = sun.norm()
    unit = sun / length
    out = {"images": torch.zeros_like(s["images"], dtype=torch.float64), "loss": torch.zeros(1, dtype=torch.float64).cuda(),
           "palette": torch.zeros_like(palette), "albedo": torch.zeros_like(albedo), "sun": torch.zeros_like(sun)}
    w, h = case["width"], case["height"]
    for v, cam in enumerate(s["cams"]):
        rec = s["hits"][v].cpu().numpy().view(vt.HIT_DTYPE).reshape(-1)
        got = torch.from_numpy(np.flatnonzero(rec["flags"] & vt.HIT_PRIMARY)).cuda()
        hit = rec[got.cpu().numpy()]
        cell = torch.from_numpy(hit["voxel"].astype(np.int64)).cuda()
        mat = torch.from_numpy(hit["material"].astype(np.int64)).cuda()
        face = torch.from_numpy(hit["face"].astype(np.int64)).cuda()
        t = torch.from_numpy(hit["t"].astype(np.float64)).cuda()
        view = torch.tensor(list(cam.view), dtype=torch.float64).cuda().reshape(4, 4)[:, :3]
        u = ((got % w).double() / w * 2.0 - 1.0) * cam.tan_half_fov
        e = (torch.div(got, w, rounding_mode="floor").double() / h * 2.0 - 1.0) * (h / w) * cam.tan_half_fov
        d = u[:, None] * view[0] + e[:, None] * view[1] + view[2] + view[3]
        d = d / d.norm(dim=1, keepdim=True)
        n = torch.zeros_like(d)
        n.scatter_(1, (face >> 1)[:, None], torch.where((face & 1) == 0, -1.0, 1.0).double()[:, None])
        o = torch.tensor(list(cam.pos)[:3], dtype=torch.float64).cuda() + d * t[:, None] + 0.001 * n
        lit = ~_blocked(solid, o, torch.where(sun == 0, 0.001, sun).expand_as(o), 512)
        facing = n @ unit
        shade = ambient + diffuse * facing.clamp(min=0) * lit
        image = out["images"][v].view(-1, 3)
        image[got] = palette[mat] * albedo[cell, None] * shade[:, None]
        off = image - s["targets"][v].view(-1, 3).double()
        out["loss"] += (off * off).sum()
        g = 2.0 * off[got]
        out["palette"].index_add_(0, mat, g * (albedo[cell] * shade)[:, None])
        out["albedo"].index_add_(0, cell, (g * palette[mat]).sum(1) * shade)
        k = (g * palette[mat]).sum(1) * albedo[cell] * diffuse * (lit & (facing > 0)) / length
        out["sun"] += (k[:, None] * (n - facing[:, None] * unit)).sum(0)
    return out
