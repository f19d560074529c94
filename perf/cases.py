"""Workloads of the volume raycaster, each run through the calls a program
makes: a view of a volume in each storage form, a multi-pane frame, section
scrolling, a flattened segment, a differentiable training step, opening a
volume, and the streamed cache.

`listed()` names twelve of them, `draw()` gives others of the same ranges.
A case is a dict with a "kind" and its sizes and options:

  cube     one view of a whole-volume cube with mips (Context.raycast)
  bricks   one view of the LOD brick cache, optionally with overlay atlases
  frame    one frame of the headless renderer, read back to pinned memory
  panes    a perspective pane and three slice panes of the brick cache, one
           call
  shard    one view of a single-level brick atlas
  slab     the tiled slab scrolls by one slice, then one view
  clip     the clipmap's window scrolls by one slice, then one view
  vslab    the virtual slab scrolls by one slice, then one view
  surf     a flattened window is baked, then viewed
  diff     forward, loss gradient and adjoint of a batch of small views
  open     a volume becomes a brick cache, a cube or an atlas, and its first
           view is drawn
  stream   the residency pump runs for a moved camera, then one view
"""
import math
import random

import numpy as np
import torch

import render3d_b200 as rb

CUTOFF = 0.99

MODES = {"full": rb.MODE_FULL, "flat": rb.MODE_FLAT, "mip": rb.MODE_MIP,
         "depth": rb.MODE_DEPTH, "heat": rb.MODE_HEATMAP}


def listed():
    return [
        # a thumbnail: the smallest call, launch latency
        {"name": "cube_thumb", "kind": "cube", "nx": 96, "ny": 96, "nz": 96, "w": 128, "h": 96,
         "mode": "full", "fast": False, "mips": True},
        # the small configuration: a 256^3 cube, full shading, no LOD
        {"name": "cube_256", "kind": "cube", "nx": 256, "ny": 256, "nz": 256, "w": 512, "h": 512,
         "mode": "full", "fast": False, "mips": False},
        # the headline: a frame of the 1024^3 orbit with its read-back
        {"name": "frame_1024", "kind": "frame", "nx": 1024, "ny": 1024, "nz": 1024, "w": 1920,
         "h": 1080, "mode": "full", "fast": False, "overlay": 0},
        # the same volume as a maximum projection
        {"name": "bricks_1024_mip", "kind": "bricks", "nx": 1024, "ny": 1024, "nz": 1024,
         "w": 1920, "h": 1080, "mode": "mip", "fast": False, "overlay": 0},
        # four panes of an odd-sized volume in an odd-sized window
        {"name": "panes_odd", "kind": "panes", "nx": 700, "ny": 523, "nz": 611, "w": 1597,
         "h": 901, "mode": "full", "fast": False},
        # a shard opened without its LOD tree
        {"name": "shard_512", "kind": "shard", "nx": 512, "ny": 512, "nz": 512, "w": 1280,
         "h": 720, "mode": "full", "fast": False},
        # paging through the slices of a wide section
        {"name": "slab_4096", "kind": "slab", "nx": 4096, "ny": 4096, "nz": 48, "w": 1920,
         "h": 1080, "mode": "full", "fast": False, "depth": 30},
        {"name": "vslab_4000", "kind": "vslab", "nx": 4000, "ny": 3500, "nz": 64, "w": 1600,
         "h": 900, "mode": "full", "fast": False, "depth": 24},
        # panning a flattened segment
        {"name": "surf_1536", "kind": "surf", "nx": 768, "ny": 768, "nz": 768, "w": 1600,
         "h": 900, "mode": "full", "win": 1536, "layers": 80, "pitch": 0.5},
        # one training step of the differentiable configuration
        {"name": "train_256", "kind": "diff", "nx": 256, "ny": 256, "nz": 256, "views": 64,
         "w": 256, "h": 256, "step": 0.5, "tape": True, "det": True, "ckpt": 64, "faint": False},
        # a small odd step without a tape, float atomics, every sample lit
        {"name": "train_odd", "kind": "diff", "nx": 97, "ny": 90, "nz": 101, "views": 5,
         "w": 151, "h": 117, "step": 0.5, "tape": False, "det": False, "ckpt": 32, "faint": True},
        # opening the headline's volume: pyramid, page table, slots, first view
        {"name": "open_1024", "kind": "open", "form": "bricks", "nx": 1024, "ny": 1024,
         "nz": 1024, "w": 960, "h": 540, "mode": "flat", "fast": False, "filter": 0},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cube", "bricks", "bricks", "frame", "panes", "shard", "slab", "clip",
                       "vslab", "surf", "diff", "diff", "open", "open", "stream"])
    w = _spread(rng, 96, 1920)
    c = {"kind": kind, "w": w, "h": max(40, min(1080, int(w * rng.uniform(0.5, 0.8))))}
    edge = _spread(rng, 64, 900)
    c["nx"], c["ny"], c["nz"] = (max(33, int(edge * rng.uniform(0.7, 1.0))) for _ in range(3))
    c["fast"] = rng.random() < 0.25
    c["mode"] = rng.choice(["full", "full", "full", "flat", "mip", "depth", "heat"])
    if kind == "cube":
        for a in ("nx", "ny", "nz"):
            c[a] = min(c[a], 400)
        c["mips"] = rng.random() < 0.6
        c["w"], c["h"] = min(c["w"], 1024), min(c["h"], 640)
    elif kind in ("bricks", "frame"):
        c["overlay"] = rng.choice([0, 0, 0, 1, 17, 4])
        if kind == "frame" or c["mode"] in ("depth", "heat"):
            c["overlay"] = 0
    elif kind == "panes":
        c["mode"] = rng.choice(["full", "mip", "flat"])
    elif kind == "shard":
        c["nx"] = c["ny"] = c["nz"] = 128 * rng.randint(1, 4)
        c["w"], c["h"] = min(c["w"], 1280), min(c["h"], 720)
    elif kind in ("slab", "clip", "vslab"):
        c["nx"], c["ny"] = _spread(rng, 1100, 4096), _spread(rng, 1100, 4096)
        c["depth"] = rng.randint(6, 30)
        c["nz"] = c["depth"] + rng.randint(8, 20)
        c["mode"] = rng.choice(["full", "full", "flat", "mip"])
    elif kind == "surf":
        c["nx"] = c["ny"] = c["nz"] = max(200, min(edge, 768))
        c["win"], c["layers"] = _spread(rng, 200, 1536), rng.randint(9, 80)
        c["pitch"] = rng.choice([0.5, 1.0, 2.0])
        c["mode"] = rng.choice(["full", "flat", "mip"])
    elif kind == "diff":
        del c["mode"], c["fast"]
        big = _spread(rng, 40, 256)
        c["nx"], c["ny"], c["nz"] = (max(17, int(big * rng.uniform(0.8, 1.0))) for _ in range(3))
        c["w"], c["h"] = _spread(rng, 33, 256), _spread(rng, 33, 256)
        c["views"] = _spread(rng, 1, 48)
        c["step"] = rng.choice([0.5, 1.0])
        c["tape"], c["det"] = rng.random() < 0.6, rng.random() < 0.5
        c["ckpt"] = rng.choice([32, 64, 128])
        c["faint"] = rng.random() < 0.3
    elif kind == "open":
        c["form"] = rng.choice(["bricks", "bricks", "cube", "shard"])
        if c["form"] == "shard":
            c["nx"] = c["ny"] = c["nz"] = 128 * rng.randint(1, 4)
        c["filter"] = rng.choice([0, 0, 1, 2, 3, 4, 256]) if c["form"] == "bricks" else 0
        c["mode"] = rng.choice(["flat", "full"])
        c["w"], c["h"] = min(c["w"], 960), min(c["h"], 540)
    elif kind == "stream":
        for a in ("nx", "ny", "nz"):
            c[a] = max(c[a], 200) // 2 + 100
        c["budget"] = rng.randint(1, 16)
    return c


# ------------------------------------------------------------------ inputs

def _levels(c):
    n, lev = max(c["nx"], c["ny"], c["nz"]), 1
    while lev < 4 and n > (128 << (lev - 1)):
        lev += 1
    return lev


def _context(c, lut):
    ctx = rb.Context(0)
    ctx.set_transfer(lut)
    ctx.set_alpha_cutoff(CUTOFF)
    if c.get("fast"):
        ctx.set_quality(rb.QUALITY_FAST)
    return ctx


def _orbit(c, lut, seed, shape, i=0):
    """A view of the scripted orbit at a phase of the seed's."""
    m = float(max(shape))
    target = tuple(0.5 * s / m for s in shape)
    phase = random.Random(seed * 31 + i).random()
    return rb.orbit_view(phase, c["w"], c["h"], lut, target=target, step_voxels=0.5,
                         mode=MODES[c["mode"]], frame_index=i)


def _section_view(c, lut, i, phase):
    """A camera facing a wide section, a little off its normal."""
    nx, ny = c["nx"], c["ny"]
    ext = (1.0, ny / nx, c["depth"] / nx)
    return rb.camera_view(0.05 * math.sin(i * 0.05 + phase), 0.02, 0.16, c["w"], c["h"], lut,
                          target=(0.3 + 0.4 * phase, 0.5 * ext[1], 0.5 * ext[2]),
                          step_voxels=0.5, mode=MODES[c["mode"]], frame_index=i)


def _slice_pane(c, lut, shape, axis, w, h, org, brick_mode, rng):
    """An orthographic pane of 32 slices across `axis` (0 z, 1 x, 2 y)."""
    m = float(max(shape))
    ext = [s / m for s in shape]
    a = {0: 2, 1: 0, 2: 1}[axis]
    u, v = [k for k in range(3) if k != a]
    p = rb.camera_view(0.0, 0.0, 1.0, w, h, lut, step_voxels=0.5, mode=MODES[c["mode"]])
    o, f, r, up = [0.5 * e for e in ext], [0.0] * 3, [0.0] * 3, [0.0] * 3
    o[a], f[a] = -0.5, 1.0
    half = 0.5 * max(ext[v], ext[u] * h / w)
    r[u], up[v] = half * w / h, half
    p.cam_origin[:], p.cam_forward[:], p.cam_right[:], p.cam_up[:] = o, f, r, up
    p.view_flags = rb.VIEW_ORTHO | rb.VIEW_AXIS(axis)
    p.slab_z0, p.slab_depth = float(rng.randint(0, max(0, shape[a] - 33))), min(32, shape[a])
    p.brick_mode = brick_mode
    p.view_org = org[0] | (org[1] << 16)
    return p


def _sheet(n):
    """A wavy 257 x 257 sheet through the middle of an n^3 volume."""
    g = 257
    d = 0.7 * n / (g - 1)
    j, i = np.mgrid[0:g, 0:g].astype(np.float64)
    x, y = 0.15 * n + d * i, 0.15 * n + d * j
    ax, ay, kx, ky = 0.06 * n, 0.04 * n, 11.0 / n, 8.0 / n
    z = 0.5 * n + ax * np.sin(x * kx) + ay * np.cos(y * ky)
    nrm = np.stack([-ax * kx * np.cos(x * kx), ay * ky * np.sin(y * ky), np.ones_like(x)], -1)
    nrm /= np.linalg.norm(nrm, axis=-1, keepdims=True)
    coords = np.ones((g, g, 4), np.float32)
    coords[..., 0], coords[..., 1], coords[..., 2] = x, y, z
    normals = np.zeros((g, g, 4), np.float32)
    normals[..., :3] = nrm
    return coords, normals, 1.0 / d


def _diff_inputs(c, seed):
    """Density, TF, views, target and step options of a training step."""
    lut8 = rb.scroll_ramp_tf()
    if c["faint"]:  # every sample contributes a little
        lut8 = rb.tf_build([(0, (20, 30, 40, 6)), (255, (220, 210, 200, 40))])
    lut = torch.tensor(lut8.astype(np.float32) / 255.0, device="cuda")
    ctx = _context(c, lut8)
    vol = ctx.phantom((c["nx"], c["ny"], c["nz"]), seed=seed)
    clean = vol.float() / 255.0
    g = torch.Generator(device="cuda").manual_seed(seed)
    dens = clean + torch.randn(clean.shape, device="cuda", generator=g) * (10.0 / 255.0)
    views = []
    for i in range(c["views"]):
        p = rb.orbit_view((i + random.Random(seed).random()) / c["views"], c["w"], c["h"], lut8,
                          step_voxels=c["step"], frame_index=i)
        p.max_mip = 0.0
        views.append(p)
    return ctx, lut, clean, dens, views


def prepare(case, seed):
    c, kind = case, case["kind"]
    rng = random.Random(seed)
    lut = rb.scroll_ramp_tf()
    shape = (c["nx"], c["ny"], c["nz"])
    s = {"case": c}
    if kind == "diff":
        ctx, tf, clean, dens, views = _diff_inputs(c, seed)
        n = c["views"] * c["w"] * c["h"] * 3
        s.update(ctx=ctx, tf=tf, dens=dens, views=views,
                 stream=torch.cuda.ExternalStream(ctx.stream),
                 target=torch.empty(n, device="cuda"), rgb=torch.empty(n, device="cuda"),
                 grad=torch.empty(n, device="cuda"), g_dens=torch.empty_like(dens),
                 g_lut=torch.empty_like(tf), g_scale=torch.empty(1, device="cuda"))
        torch.cuda.synchronize()
        ctx.diff_forward(clean, tf, views, s["target"], stream=ctx.stream)
        torch.cuda.synchronize()
        return s
    if kind == "frame":
        tmp = rb.Context(0)
        vol = tmp.phantom(shape, seed=seed)
        r = rb.Renderer(c["w"], c["h"])
        r.bricks_begin_volume(vol, _levels(c))
        tmp.close()
        r.set_transfer(lut)
        r.set_alpha_cutoff(CUTOFF)
        if c["fast"]:
            r.set_quality(rb.QUALITY_FAST)
        p = _orbit(c, lut, seed, shape)
        r.bricks_params(p)
        s.update(renderer=r, view=p,
                 out=torch.empty((c["h"], c["w"], 4), dtype=torch.uint8, pin_memory=True))
        torch.cuda.synchronize()
        return s
    ctx = _context(c, lut)
    vol = ctx.phantom(shape, seed=seed)
    img = torch.zeros((c["h"], c["w"], 4), dtype=torch.uint8, device="cuda")
    s.update(ctx=ctx, img=img)
    if kind == "cube":
        ctx.upload_volume(vol)
        p = _orbit(c, lut, seed, shape)
        p.max_mip = 10.0 if c["mips"] else 0.0
        s["views"] = [p]
    elif kind in ("bricks", "panes"):
        ctx.bricks_build(vol, _levels(c))
        p = _orbit(c, lut, seed, shape)
        p.brick_mode = ctx.brick_mode
        s["views"] = [p]
        if kind == "panes":
            w0, h0 = c["w"] // 2, c["h"] // 2
            p.viewport[0], p.viewport[1] = w0, h0
            for axis, (ox, oy) in enumerate(((w0, 0), (0, h0), (w0, h0))):
                s["views"].append(_slice_pane(
                    c, lut, shape, axis, c["w"] - w0 if ox else w0, c["h"] - h0 if oy else h0,
                    (ox, oy), ctx.brick_mode, rng))
        elif c["overlay"]:
            for k, bit in enumerate((1, 4, 8, 16)):
                if c["overlay"] & bit:
                    ctx.overlay_build(k, ctx.phantom(shape, seed=seed + 7 + k))
            p.overlay_flags, p.overlay_gain = c["overlay"] | (128 << 16), 1.5
    elif kind == "shard":
        ctx.shard_build(vol)
        p = _orbit(c, lut, seed, shape)
        p.brick_mode = ctx.shard_mode
        s["views"] = [p]
    elif kind in ("slab", "clip", "vslab"):
        s["z"], s["dz"], s["phase"] = 0, 1, rng.random()
        if kind == "slab":
            ctx.slab_build(vol, c["depth"] + 2, 0)
        elif kind == "clip":
            ctx.clip_build(vol, c["depth"])
        else:
            ctx.vslab_begin(vol, c["nx"], c["ny"], c["depth"])
            for _ in range(12):
                ctx.vslab_frame(c["nx"] / 2, c["ny"] / 2, 0, 64)
        s["view"] = _section_view(c, lut, 0, s["phase"])
    elif kind == "surf":
        ctx.bricks_build(vol, _levels(c))
        coords, normals, cells = _sheet(c["nx"])
        ctx.surf_begin(coords, normals)
        ctx.surfvol_begin(c["win"], c["win"], c["layers"], c["layers"] // 2, cells, cells)
        p = rb.FrameParams()
        p.viewport[0], p.viewport[1] = c["w"], c["h"]
        p.mode = MODES[c["mode"]]
        span = c["win"] * c["pitch"]
        p.cam_origin[:] = (0.5 * span, 0.5 * span, 0.0)
        p.cam_right[:] = (0.4 * span, 0.0, 0.0)
        p.cam_up[:] = (0.0, 0.4 * span * c["h"] / c["w"], 0.0)
        p.step_voxels, p.density, p.threshold = 0.5, 1.5, 0.02
        p.slab_z0, p.slab_depth = 0.0, max(1, (2 * c["layers"]) // 3)
        s["view"], s["u0"] = p, rng.uniform(0.0, 0.05 * span)
    elif kind == "open":
        s["vol"] = vol
        s["views"] = [_orbit(c, lut, seed, shape)]
        ctx.bricks_postfilter(c["filter"], 0.6)
    elif kind == "stream":
        lev = _levels(c)
        nb = [-(-n // 128) for n in shape]
        ctx.stream_begin(vol, lev, max(8, nb[0] * nb[1] * nb[2] // 2))
        s["views"] = [_orbit(c, lut, seed, shape, i) for i in range(4)]
        s["at"] = 0
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------- passes

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "diff":
        ctx, st = state["ctx"], state
        ctx.diff_forward(st["dens"], st["tf"], st["views"], st["rgb"], stream=ctx.stream,
                         tape=c["tape"])
        with torch.cuda.stream(st["stream"]):
            torch.sub(st["rgb"], st["target"], out=st["grad"])
        ctx.raycast_bwd(st["dens"], st["tf"], st["views"], st["grad"], st["g_dens"], st["g_lut"],
                        st["g_scale"], c["ckpt"], c["det"], stream=ctx.stream, tape=c["tape"])
        return {"rgb": st["rgb"], "density": st["g_dens"], "lut": st["g_lut"],
                "scale": st["g_scale"]}
    if kind == "frame":
        r = state["renderer"]
        r.frame(state["view"])
        return r.read_frame(state["out"])
    ctx, img = state["ctx"], state["img"]
    if kind in ("slab", "clip", "vslab"):
        # the window moves one slice a pass, back and forth over the volume
        top = c["nz"] - c["depth"] - 4
        z = state["z"] + state["dz"]
        if z < 0 or z > top:
            state["dz"] = -state["dz"]
            z = state["z"] + state["dz"]
        state["z"] = z
        p = state["view"]
        if kind == "slab":
            ctx.slab_window(z)
            ctx.slab_params(p)
        elif kind == "clip":
            ctx.clip_frame(0.5 * c["nx"], 0.5 * c["ny"], z)
            ctx.clip_params(p)
        else:
            ctx.vslab_frame(0.5 * c["nx"], 0.5 * c["ny"], z, 64)
            ctx.vslab_params(p)
        p.slab_depth = c["depth"]
        p.density = 6.0
        return ctx.raycast(p, c["w"], c["h"], out=img)
    if kind == "surf":
        p = state["view"]
        ctx.surfvol_window(state["u0"], 0.0, c["pitch"], 0.0)
        ctx.surfvol_params(p)
        return ctx.raycast(p, c["w"], c["h"], out=img)
    if kind == "open":
        p, page = state["views"][0], None
        if c["form"] == "bricks":
            ctx.bricks_build(state["vol"], _levels(c))
            p.brick_mode = ctx.brick_mode
            page = ctx.bricks_read(slots=False)[0].view(np.int32)
        elif c["form"] == "shard":
            ctx.shard_build(state["vol"])
            p.brick_mode = ctx.shard_mode
        else:
            ctx.upload_volume(state["vol"])
        ctx.raycast(p, c["w"], c["h"], out=img)
        return img if page is None else [img, page]
    if kind == "stream":
        p = state["views"][state["at"]]
        state["at"] = (state["at"] + 1) % len(state["views"])
        p.brick_mode = ctx.brick_mode
        st = ctx.stream_update(p, c["budget"])
        ctx.raycast(p, c["w"], c["h"], out=img)
        return [img, st["desired"], st["uploaded"], st["resident"]]
    return ctx.raycast(state["views"], c["w"], c["h"], out=img)


def work(case):
    """Bytes: the voxels that the pass has to see once (at most the volume's,
    at most eight a sample) and its image or gradients; flops: the samples
    (a typical number a ray for the kind) times a trilinear lookup, a TF
    lookup and the compositing."""
    c, kind = case, case["kind"]
    nvox = c["nx"] * c["ny"] * c["nz"]
    if kind == "diff":
        rays = c["views"] * c["w"] * c["h"]
        samples = rays * 0.6 * max(c["nx"], c["ny"], c["nz"]) / c["step"]
        return {"bytes": 4.0 * nvox * 2 + 12.0 * rays * 3 + 8192, "flops": samples * 40.0}
    rays = c["w"] * c["h"]
    m = max(c["nx"], c["ny"], c["nz"])
    per_ray = {"bricks": 15, "frame": 15, "panes": 25, "stream": 15, "cube": 0.5 * m, "shard": 0.5 * m,
               "slab": 60, "clip": 60, "vslab": 60, "surf": c.get("layers", 0), "open": 15}[kind]
    samples = rays * per_ray
    nbytes = min(nvox, 8.0 * samples) + 4.0 * rays
    if kind == "open":
        nbytes = nvox * (2.0 + 1.0 / 7.0) + 4.0 * rays
    elif kind == "surf":
        nbytes = 2.0 * c["win"] * c["win"] * c["layers"] + 4.0 * rays
        samples += c["win"] * c["win"] * c["layers"]
    return {"bytes": float(nbytes), "flops": 30.0 * samples}


# ------------------------------------------------------------- 64-bit values

def exact(case, seed):
    """A training step in 64 bits with plain torch; images are whole numbers
    and have none."""
    c = case
    if c["kind"] != "diff":
        return None
    ctx, tf, clean, dens, views = _diff_inputs(c, seed)
    ctx.close()
    f64 = dict(dtype=torch.float64, device="cuda")
    lut = tf.double().requires_grad_(True)
    d = dens.double().reshape(-1).requires_grad_(True)
    scale = torch.tensor(float(views[0].density), **f64).requires_grad_(True)
    rgb = []
    for i, p in enumerate(views):
        with torch.no_grad():
            want = _render64(c, p, clean.double().reshape(-1), lut, scale)
        got = _render64(c, p, d, lut, scale)
        # the loss 0.5 |rgb - target|^2, whose gradient the step hands back
        (0.5 * (got - want).square().sum()).backward()
        rgb.append(got.detach().reshape(-1))
    return {"rgb": torch.cat(rgb), "density": d.grad.reshape(dens.shape), "lut": lut.grad,
            "scale": scale.grad.reshape(1)}


def _hash(px, py, frame):
    mask = 0xFFFFFFFF
    h = (px * 374761393 + py * 668265263 + (frame * 2246822519 & mask)) & mask
    h = h ^ (h >> 13)
    lo, hi = h & 0xFFFF, h >> 16
    h = (lo * 1274126177 + ((hi * 1274126177 & 0xFFFF) << 16)) & mask
    return (h >> 8).double() / 16777216.0


def _render64(c, p, dens, lut, scale):
    """FLAT compositing of one view over a flat density grid, (rays, 3)."""
    f64 = dict(dtype=torch.float64, device="cuda")
    w, h, n = c["w"], c["h"], (c["nx"], c["ny"], c["nz"])
    vec = lambda a: torch.tensor(list(a), **f64)  # noqa: E731
    py, px = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"),
                            indexing="ij")
    px, py = px.reshape(-1), py.reshape(-1)
    x = (px.double() + 0.5) / w * 2 - 1
    y = 1 - (py.double() + 0.5) / h * 2
    dr = vec(p.cam_forward) + x[:, None] * vec(p.cam_right) + y[:, None] * vec(p.cam_up)
    dr = dr / dr.norm(dim=1, keepdim=True)
    rot = torch.stack([vec(p.vol_r0), vec(p.vol_r1), vec(p.vol_r2)])
    dr = dr @ rot
    ro = (vec(p.cam_origin) - vec((p.vol_tx, p.vol_ty, p.vol_tz)) - 0.5) @ rot + 0.5
    t0, t1 = -ro / dr, (1 - ro) / dr
    tn = torch.minimum(t0, t1).amax(1).clamp(min=0.0)
    tf = torch.maximum(t0, t1).amin(1)
    dt = float(p.step_voxels) / max(n)
    t = tn + _hash(px, py, int(p.frame_index)) * dt
    span = ((tf - tn) / (4096 * dt)).clamp(min=1.0)
    count = torch.where(tn < tf, ((tf - t) / (dt * span)).ceil(), torch.zeros_like(t))
    steps = int(count.max().clamp(min=1, max=4096))
    rows = torch.arange(w * h, device="cuda")
    size = torch.tensor(n, **f64)

    def sample(ray, at):
        pos = ro + at[..., None] * dr[ray]
        tc = torch.minimum((pos * size - 0.5).clamp(min=0.0), size - 1)
        i0 = tc.floor()
        fr = tc - i0
        i0 = i0.long()
        i1 = torch.minimum(i0 + 1, size.long() - 1)
        v = 0.0
        for k in range(8):
            b = [(k >> a) & 1 for a in range(3)]
            q = [i1[..., a] if b[a] else i0[..., a] for a in range(3)]
            wt = 1.0
            for a in range(3):
                wt = wt * (fr[..., a] if b[a] else 1 - fr[..., a])
            v = v + wt * dens[(q[2] * n[1] + q[1]) * n[0] + q[0]]
        tt = (v * 256 - 0.5).clamp(0.0, 255.0)
        j0 = tt.detach().floor().long()
        f = tt - j0
        s = lut[j0] * (1 - f)[..., None] + lut[(j0 + 1).clamp(max=255)] * f[..., None]
        alpha = s[..., 3].clamp(0.0, 1.0)
        a = 1 - (1 - alpha) ** (scale * float(p.step_voxels) * span[ray])
        keep = (a.detach() > 0.003) & (v.detach() >= float(p.threshold))
        return s[..., :3], torch.where(keep, a, torch.zeros_like(a)), keep

    # the contributing samples of every ray, found without gradients
    lists, depth = [], 1
    with torch.no_grad():
        for part in rows.split(max(1, 16_000_000 // steps)):
            k = torch.arange(steps, device="cuda")
            at = t[part, None] + k * (dt * span[part, None])
            _, a, keep = sample(part[:, None].expand(-1, steps), at)
            live = k < count[part, None]
            a, keep = torch.where(live, a, torch.zeros_like(a)), keep & live
            before = torch.cat([torch.zeros_like(a[:, :1]), 1 - (1 - a).cumprod(1)[:, :-1]], 1)
            keep = keep & (before < CUTOFF)
            rank = keep.cumsum(1) - 1
            m = int(keep.sum(1).max())
            depth = max(depth, m)
            chosen = torch.full((len(part), max(m, 1)), -1, dtype=torch.long, device="cuda")
            r, q = keep.nonzero(as_tuple=True)
            chosen[r, rank[r, q]] = q
            lists.append(chosen)
    chosen = torch.cat([torch.nn.functional.pad(x, (0, depth - x.shape[1]), value=-1)
                        for x in lists])
    have = chosen >= 0
    at = t[:, None] + chosen.clamp(min=0) * (dt * span[:, None])
    col, a, _ = sample(rows[:, None].expand(-1, depth), at)
    a = torch.where(have, a, torch.zeros_like(a))
    trans = torch.cat([torch.ones_like(a[:, :1]), (1 - a).cumprod(1)], 1)
    out = ((trans[:, :-1] * a)[..., None] * col).sum(1)
    return out + trans[:, -1:] * torch.tensor([0.02, 0.02, 0.03], **f64)
