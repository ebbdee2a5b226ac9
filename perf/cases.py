"""Workloads of the SH9 lightmap bake for timing it: what a program does with
this library, through its public entry points, over the range of sizes.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what the program holds before the call
  run(state)           one pass, and its outputs
  work(case)           bytes and floating-point operations it cannot do without
  exact(case, seed)    the outputs in 64 bits, where they have such a value

A case is a dict of plain values.  "op" says which call it is:

  lightmap  bake_lightmap from a host scene (upload, BVH, raster, bake,
            masks, downsample, dilation, read-back): the command line's job
  bake      BVH build and BakeSHLightMap over a resident G-buffer, the region
            the reference times as its bake
  batch     many small independent bakes in one call
  adjoint   bake and gradient of a loss through it (torch.autograd)
  rays      FindOcclusion: closest-hit queries against a resident scene
  post      downsample, validity mask and dilation of a baked texture
  save      SaveSHLightMap to EXR files
"""
from __future__ import annotations

import ctypes as C
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from sh_baker_b200 import _capi as A
from sh_baker_b200 import api, scenes
from sh_baker_b200.autograd import bake_sh
from sh_baker_b200.scene import SPOT, Light, Material, Texture


def listed():
    return [
        # The smallest job: a quad's 64^2 lightmap, where launches and waits count.
        dict(name="lightmap_quad", op="lightmap", scene="quad", boxes=0, width=64, height=64, ss=1, spp=16, bounces=1,
             nls=1, dilation=4),
        # An ordinary job from host data: a furnished room, ragged page size.
        dict(name="lightmap_room", op="lightmap", scene="room", boxes=100, width=250, height=190, ss=2, spp=32,
             bounces=3, nls=1, dilation=16),
        # A draft of a large scene (263k triangles): upload and BVH weigh as much as the paths.
        dict(name="lightmap_atrium", op="lightmap", scene="atrium", boxes=0, width=320, height=320, ss=2, spp=16,
             bounces=3, nls=1, dilation=4),
        # The benchmark's unit quad at its own size: no ray hits anything.
        dict(name="bake_quad", op="bake", scene="quad", boxes=0, width=256, height=256, ss=1, spp=64, bounces=3,
             nls=1),
        # The benchmark's room (2,412 triangles, 5 lights) at a quarter of its page.
        dict(name="bake_room", op="bake", scene="room", boxes=200, width=512, height=512, ss=2, spp=64, bounces=3,
             nls=1),
        # The benchmark's atrium (24 lights, 15 of them emissive panels): the largest.
        dict(name="bake_atrium", op="bake", scene="atrium", boxes=0, width=768, height=768, ss=3, spp=64, bounces=4,
             nls=1),
        # Textured cut-outs and emitters, a spot light and two light samples: branching paths, odd size.
        dict(name="bake_leaves", op="bake", scene="leaves", boxes=60, width=317, height=211, ss=2, spp=32, bounces=2,
             nls=2),
        # Many small rooms at once, as for the props of a level.
        dict(name="batch_rooms", op="batch", scene="room", boxes=120, width=192, height=192, ss=1, spp=32, bounces=3,
             nls=1, bakes=16),
        # One step of fitting materials and lights to a target lightmap.
        dict(name="adjoint_room", op="adjoint", scene="room", boxes=200, width=256, height=256, ss=2, spp=32,
             bounces=3, nls=1),
        # Visibility queries of a tool against a large scene.
        dict(name="rays_atrium", op="rays", scene="atrium", boxes=0, count=2_000_003),
        # What follows a bake: 3072^2 texels down to 1024^2, gutters filled.
        dict(name="post_1024", op="post", width=1024, height=1024, ss=3, dilation=16),
        # The lightmap's file.
        dict(name="save_512", op="save", width=512, height=512, mode=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# Paths x vertices of a drawn bake stay below the largest listed bake's.
_MOST_VERTICES = 768 * 768 * 9 * 64 * 5 // 4


def draw(rng):
    op = rng.choice(["lightmap", "lightmap", "bake", "bake", "bake", "batch", "adjoint", "rays", "post", "save"])
    if op == "post":
        ss = rng.choice([1, 2, 2, 3, 4])
        top = 3072 // ss
        return dict(op=op, width=_log(rng, 33, top), height=_log(rng, 33, top), ss=ss, dilation=_log(rng, 1, 32))
    if op == "save":
        return dict(op=op, width=_log(rng, 17, 512), height=_log(rng, 17, 512), mode=rng.choice([0, 0, 1, 2]))
    if op == "rays":
        kind = rng.choice(["room", "room", "atrium", "leaves"])
        return dict(op=op, scene=kind, boxes=_log(rng, 8, 320) if kind != "atrium" else 0,
                    count=_log(rng, 1_000, 2_000_000))
    if op == "batch":
        return dict(op=op, scene="room", boxes=_log(rng, 10, 300), width=_log(rng, 32, 256), height=_log(rng, 32, 256),
                    ss=1, spp=_log(rng, 8, 64), bounces=rng.randint(1, 4), nls=1, bakes=_log(rng, 2, 24))
    kind = rng.choice(["quad", "room", "room", "room", "leaves"] if op == "adjoint" else
                      ["quad", "room", "room", "atrium", "leaves"])
    c = dict(op=op, scene=kind, boxes=0 if kind in ("quad", "atrium") else _log(rng, 4, 400),
             width=_log(rng, 40, 384 if op == "adjoint" else 640), height=_log(rng, 40, 384 if op == "adjoint" else 640),
             ss=rng.choice([1, 1, 2, 3]), spp=_log(rng, 8, 128), bounces=rng.randint(0, 4), nls=rng.choice([1, 1, 1, 2]))
    while c["width"] * c["height"] * c["ss"] ** 2 * c["spp"] * (1 + c["bounces"]) * c["nls"] > _MOST_VERTICES:
        c["spp"] = max(4, c["spp"] // 2)
        c["ss"] = max(1, c["ss"] - 1)
    if op == "lightmap":
        c["dilation"] = _log(rng, 1, 32)
    return c


# ------------------------------------------------------------------ inputs --

def _leaves(seed, boxes, res):
    """A room whose materials are 64^2 textures: half of them cut-outs with
    alpha, one an emitter with a textured emission; plus a spot light."""
    sc = scenes.procedural_room(seed=seed, n_boxes=boxes, res=res)
    rng = np.random.default_rng(seed + 17)
    yy, xx = np.mgrid[0:64, 0:64]
    for i, m in enumerate(sc.materials):
        rgb = (m.albedo.pixel_data[:3] * rng.uniform(0.5, 1.0, (64, 64, 1))).astype(np.uint8)
        if i % 2 and i < 7:
            a = np.where((xx // 8 + yy // 8) % 2, 255, 0)
            a = np.where(rng.random((64, 64)) < 0.1, 128, a).astype(np.uint8)
            px = np.concatenate([rgb, a[..., None]], 2)
        else:
            px = rgb
        sc.materials[i] = Material(name=m.name, albedo=Texture(64, 64, px.shape[2], np.ascontiguousarray(px).reshape(-1)),
                                   emission_intensity=4.0 if i == 7 else 0.0)
    sc.lights.append(Light(type=SPOT, position=(0.5, 2.7, -0.5), direction=(0.0, -1.0, 0.0), intensity=30.0))
    scenes.mark_area_lights(sc)
    return sc


def _scene(case, seed):
    kind, res = case["scene"], max(case.get("width", 512), case.get("height", 512))
    if kind == "atrium":
        return scenes.atrium(seed=seed, res=res)
    if kind == "room":
        return scenes.procedural_room(seed=seed, n_boxes=case["boxes"], res=res)
    if kind == "leaves":
        return _leaves(seed, case["boxes"], res)
    sc = scenes.unit_quad()
    rng = np.random.default_rng(seed)
    d = np.array([rng.uniform(-0.5, 0.5), -1.0, rng.uniform(-0.5, 0.5)])
    d = d / np.linalg.norm(d)
    sc.lights[0].direction = tuple(float(x) for x in d)
    sc.lights[1].position = (float(rng.uniform(-0.4, 0.4)), float(rng.uniform(0.6, 1.2)), float(rng.uniform(-0.4, 0.4)))
    sc.lights[1].intensity = float(rng.uniform(5.0, 15.0))
    return sc


def _bake_seed(seed):
    return (seed * 2654435761 + 1) & 0x7FFFFFFF


def _bake(ctx, case, seed, k=0):
    """A resident scene with its G-buffer, the config and output textures."""
    ds = api.DeviceScene(ctx, _scene(case, seed))
    rc = api.RasterConfig(case["width"], case["height"], case["ss"])
    g = api.rasterize_to_device(ds, rc)
    cfg = api.BakeConfig(samples=case["spp"], bounces=case["bounces"], num_light_samples=case["nls"],
                         seed=_bake_seed(seed))
    n = g.width * g.height
    out = (torch.empty(n * 27, dtype=torch.float32, device="cuda"), torch.empty(n, dtype=torch.float32, device="cuda"))
    return api.BatchBake(ds, g, rc, cfg), out


def _rays(case, seed):
    """Segments and half-lines from points inside the scene."""
    half = (18.0, 9.5, 13.0) if case["scene"] == "atrium" else (4.9, 2.9, 4.9)
    gen = torch.Generator("cuda").manual_seed(seed)
    n = case["count"]
    u = torch.rand((n, 8), generator=gen, device="cuda")
    r = torch.empty((n, 8), device="cuda")
    r[:, 0] = (2 * u[:, 0] - 1) * half[0]
    r[:, 1] = 0.05 + u[:, 1] * half[1]
    r[:, 2] = (2 * u[:, 2] - 1) * half[2]
    z, phi = 2 * u[:, 3] - 1, 2 * math.pi * u[:, 4]
    s = torch.sqrt(1 - z * z)
    r[:, 3], r[:, 4], r[:, 5] = s * torch.cos(phi), z, s * torch.sin(phi)
    r[:, 6] = 0.001
    r[:, 7] = torch.where(u[:, 5] < 0.5, torch.full_like(u[:, 6], float("inf")), 0.5 + 10 * u[:, 6])
    return r


def _texture(width, height, seed, mask_of):
    """SH and environment visibility like a bake's (smooth fields with sample
    noise) inside charts of a page, zero in the gutters and the unused rest."""
    gen = torch.Generator("cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    y = torch.arange(height, device="cuda")[:, None]
    x = torch.arange(width, device="cuda")[None, :]
    cw, ch, gap = int(rng.integers(30, 90)), int(rng.integers(30, 90)), int(rng.integers(2, 6)) * mask_of
    mask = ((x % (cw * mask_of)) < cw * mask_of - gap) & ((y % (ch * mask_of)) < ch * mask_of - gap)
    mask = (mask & (y < int(0.85 * height) + 1)).to(torch.uint8)
    f = torch.from_numpy(rng.uniform(1, 6, (27, 2))).to("cuda", torch.float32)
    sh = torch.empty((height, width, 27), device="cuda")
    for k in range(27):
        base = torch.sin(f[k, 0] * x / width + k) * torch.cos(f[k, 1] * y / height)
        sh[:, :, k] = (1.0 + base) if k < 3 else 0.3 * base
    sh *= 1.0 + 0.01 * torch.randn(sh.shape, generator=gen, device="cuda")
    env = (0.5 + 0.5 * torch.sin(3.0 * x / width) * torch.cos(2.0 * y / height)).clamp(0, 1)
    sh *= mask[:, :, None]
    return sh, (env * mask).contiguous(), mask.contiguous()


def prepare(case, seed):
    op = case["op"]
    ctx = api.default_context()
    st = {"case": case, "op": op, "ctx": ctx}
    if op == "lightmap":
        h, w = case["height"], case["width"]
        st["scene"] = _scene(case, seed)
        st["seed"] = _bake_seed(seed)
        st["out"] = tuple(torch.empty(s, dtype=t, pin_memory=True).numpy() for s, t in
                          (((h, w, 9, 3), torch.float32), ((h, w), torch.float32), ((h, w), torch.uint8)))
    elif op == "bake":
        st["bake"], st["out"] = _bake(ctx, case, seed)
    elif op == "batch":
        st["bakes"], st["outs"] = [], []
        for k in range(case["bakes"]):  # sizes around the case's, from half to all of it
            c = dict(case, boxes=max(4, case["boxes"] * (k % 4 + 1) // 4),
                     width=max(16, case["width"] * (k % 3 + 2) // 4), height=max(16, case["height"] * (k % 5 + 4) // 8))
            b, o = _bake(ctx, c, seed * 64 + k)
            st["bakes"].append(b)
            st["outs"].append(o)
    elif op == "adjoint":
        st["bake"], (sh, _) = _bake(ctx, case, seed)
        ds = st["bake"].scene
        gen = torch.Generator("cuda").manual_seed(seed)
        st["albedo"] = (0.1 + 0.8 * torch.rand((ds.n_materials, 3), generator=gen, device="cuda")).requires_grad_()
        st["light"] = (5.0 + 20.0 * torch.rand(ds.n_lights, generator=gen, device="cuda")).requires_grad_()
        st["target"] = torch.rand((sh.numel() // 27, 9, 3), generator=gen, device="cuda")
    elif op == "rays":
        st["scene"] = api.DeviceScene(ctx, _scene(case, seed))
        st["rays"] = _rays(case, seed)
        st["hits"] = torch.empty((case["count"], C.sizeof(A.Hit) // 4), dtype=torch.int32, device="cuda")
    elif op == "post":
        s = case["ss"]
        n = case["width"] * case["height"]
        st["sh"], st["env"], st["mask"] = _texture(case["width"] * s, case["height"] * s, seed, s)
        st["out"] = (torch.empty(n * 27, device="cuda"), torch.empty(n, device="cuda"),
                     torch.empty(n, dtype=torch.uint8, device="cuda"))
    elif op == "save":
        sh, env, _ = _texture(case["width"], case["height"], seed, 1)
        st["sh"] = sh.view(case["height"], case["width"], 9, 3).cpu().numpy()
        st["env"] = env.cpu().numpy()
        st["dir"] = tempfile.TemporaryDirectory()
        # the files' bytes, each in a buffer of the largest size (stored raw)
        chunks, most = (case["height"] + 15) // 16, {0: 28, 1: 4, 2: 4}[case["mode"]]
        cap = case["width"] * case["height"] * 2 * most + 16 * chunks + 4096
        st["files"] = [np.zeros(cap, np.uint8) for _ in range({0: 1, 1: 9, 2: 3}[case["mode"]])]
    return st


# -------------------------------------------------------------------- a pass --

def run(st):
    op, case, ctx = st["op"], st["case"], st["ctx"]
    if op == "lightmap":
        r = api.bake_lightmap(st["scene"], case["width"], case["height"], case["spp"], case["bounces"], case["ss"],
                              case["dilation"], st["seed"], case["nls"], ctx=ctx, out=st["out"])
        return {"sh": r.sh, "env": r.env, "mask": r.mask}
    if op == "bake":
        st["bake"].scene.rebuild_bvh()
        api.bake_plain_device(st["bake"], *st["out"])
        return {"sh": st["out"][0], "env": st["out"][1]}
    if op == "batch":
        outs, _ = api.bake_batch(ctx, st["bakes"], outputs=st["outs"])
        return outs
    if op == "adjoint":
        sh = bake_sh(st["albedo"], st["light"], st["bake"])
        loss = (sh - st["target"]).square().sum()
        d_albedo, d_light = torch.autograd.grad(loss, (st["albedo"], st["light"]))
        return {"sh": sh.detach(), "d_albedo": d_albedo, "d_light": d_light}
    if op == "rays":
        hits = st["hits"]
        A.check(ctx.lib.shb_find_occlusion(st["scene"].h, st["rays"].data_ptr(), case["count"], hits.data_ptr(), 1))
        f = hits.view(torch.float32)
        return {"position": f[:, 0:3], "uv": f[:, 3:5], "normal": f[:, 5:8], "t": f[:, 10], "material": hits[:, 8],
                "hit": hits[:, 9], "prim": hits[:, 11]}
    if op == "post":
        w, h, s, lib = case["width"], case["height"], case["ss"], ctx.lib
        sh, env, mask = st["out"]
        A.check(lib.shb_downsample(ctx.h, st["sh"].data_ptr(), w * s, h * s, 27, s, sh.data_ptr(), 1))
        A.check(lib.shb_downsample(ctx.h, st["env"].data_ptr(), w * s, h * s, 1, s, env.data_ptr(), 1))
        A.check(lib.shb_downsample_validity_mask(ctx.h, st["mask"].data_ptr(), w, h, s, mask.data_ptr(), 1))
        A.check(lib.shb_dilate(ctx.h, A.DILATE_SH9, w, h, sh.data_ptr(), mask.data_ptr(), case["dilation"], 1))
        A.check(lib.shb_dilate(ctx.h, A.DILATE_F32, w, h, env.data_ptr(), mask.data_ptr(), case["dilation"], 1))
        return {"sh": sh, "env": env, "mask": mask}
    path = Path(st["dir"].name)
    if not api.SaveSHLightMap(st["sh"], st["env"], path / "map.exr", case["mode"], ctx=ctx):
        raise RuntimeError("SaveSHLightMap failed")
    for p, buf in zip(sorted(path.glob("*.exr")), st["files"]):
        with open(p, "rb") as f:
            buf[f.readinto(buf):] = 0
    return st["files"]


# ------------------------------------------------------------------ the least --

_TRIANGLES = {"quad": 2, "atrium": 263352}


def _tris(case):
    return _TRIANGLES.get(case["scene"]) or 12 * (case["boxes"] + 1)


def _ray_flops(tris):
    """An 8-wide node per level (8 boxes of 3 slabs: 12 operations each) and a
    leaf of 4 triangles (about 40 each)."""
    levels = max(1, math.ceil(math.log(max(1, tris / 4), 8)))
    return levels * 8 * 12 + 4 * 40


def work(case):
    op = case["op"]
    if op in ("post", "save"):
        n = case["width"] * case["height"]
        if op == "save":  # 28 floats in, 28 halves through, about their bytes again in the file
            return {"bytes": n * 28 * (4 + 2), "flops": 28 * n}
        s2 = case["ss"] ** 2
        return {"bytes": n * (s2 + 1) * (28 * 4 + 1), "flops": n * s2 * 28}
    tris = _tris(case)
    geometry = tris * 3 * (12 + 12 + 8 + 8 + 16) // 2  # about two triangles per three vertices
    if op == "rays":
        return {"bytes": case["count"] * (32 + 48) + geometry, "flops": case["count"] * _ray_flops(tris)}
    # about this share of a page lies inside charts
    fill = {"quad": 1.0, "atrium": 0.25}.get(case["scene"], 0.55)
    texels = case["width"] * case["height"] * case["ss"] ** 2
    bakes = case.get("bakes", 1)
    # a path's rays: one closest hit and one light query per vertex and light
    # sample, plus the texel's own light queries; the quad's paths hit nothing
    vertices = 1 if case["scene"] == "quad" else 1 + case["bounces"]
    lights = case["nls"] * (1 if case["scene"] == "quad" else 1 + vertices)
    flops = bakes * fill * texels * case["spp"] * (vertices + lights) * _ray_flops(tris) + tris * 3 * 32 * 8
    n_bytes = bakes * (texels * (64 + 112) + geometry)
    if op == "lightmap":
        n_bytes += case["width"] * case["height"] * 113
    if op == "adjoint":
        return {"bytes": 2 * n_bytes, "flops": 2 * flops}
    return {"bytes": n_bytes, "flops": flops}


# -------------------------------------------------------------- in 64 bits ----
# A bake whose rays hit something has no such value: a light pick or a hit
# that lies within rounding of its limit sends the path elsewhere, and every
# later vertex with it.  The unit quad's paths hit nothing: its texels are
# sums over the light picks, which are computed here from the counter stream.

def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al. 2011) over uint64 arrays of 32-bit words."""
    m32 = np.uint64(0xFFFFFFFF)
    sh = np.uint64(32)
    for r in range(10):
        if r:
            k0 = (k0 + np.uint64(0x9E3779B9)) & m32
            k1 = (k1 + np.uint64(0xBB67AE85)) & m32
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> sh) ^ c1 ^ k0, p1 & m32, (p0 >> sh) ^ c3 ^ k1, p0 & m32
    return c0, c1, c2, c3


def _sh9(d):
    x, y, z = d[..., 0], d[..., 1], d[..., 2]
    return np.stack([np.full_like(x, 0.282095), 0.488603 * y, 0.488603 * z, 0.488603 * x, 1.092548 * x * y,
                     1.092548 * y * z, 0.315392 * (3 * z * z - 1), 1.092548 * x * z, 0.546274 * (x * x - y * y)], -1)


def _quad_exact(case, seed):
    sc = _scene(case, seed)
    W, H, spp, nls = case["width"] * case["ss"], case["height"] * case["ss"], case["spp"], case["nls"]
    if W * H * spp * nls > 30_000_000:
        return None
    sun, point = sc.lights
    uv = np.stack(np.meshgrid((np.arange(W) + 0.5) / W, (np.arange(H) + 0.5) / H), -1).reshape(-1, 2)
    P = np.stack([uv[:, 0] - 0.5, np.zeros(W * H), uv[:, 1] - 0.5], -1)
    to_sun = np.broadcast_to(-np.array(sun.direction, np.float64), P.shape)
    to_point = np.array(point.position, np.float64) - P
    rad = np.stack([np.full(W * H, sun.intensity), point.intensity / (to_point ** 2).sum(-1)], -1)
    total = rad.sum(-1)
    pdf = rad / total[:, None]
    y = np.stack([_sh9(to_sun), _sh9(to_point)], 1)
    value = np.where(pdf < 1e-3, 0.0, rad / (pdf * nls))[:, :, None] * y  # one pick's term, by light
    acc = np.zeros((W * H, 9))
    texel, zero = np.arange(W * H, dtype=np.uint64), np.uint64(0)
    for s in range(spp):
        for j in range(nls):
            bits = _philox(np.full(W * H, s, np.uint64), zero, np.uint64(1), np.uint64(j >> 2),
                           np.uint64(_bake_seed(seed)), texel)[j & 3]
            u = (bits >> np.uint64(8)).astype(np.float64) / 16777216.0
            acc += np.where((u * total < rad[:, 0])[:, None], value[:, 0], value[:, 1])
    sh = np.repeat((acc / spp)[:, :, None], 3, 2)
    env = np.ones(W * H)
    if case["op"] == "bake":
        return {"sh": sh.reshape(-1), "env": env}
    s = case["ss"]
    w, h = case["width"], case["height"]
    sh = sh.reshape(h, s, w, s, 9, 3).mean((1, 3))
    return {"sh": sh, "env": env.reshape(h, s, w, s).mean((1, 3)), "mask": None}


def _post_exact(case, seed):
    w, h, s = case["width"], case["height"], case["ss"]
    sh, env, mask = _texture(w * s, h * s, seed, s)
    x = torch.cat([sh, env[:, :, None]], 2).double()
    x = x.view(h, s, w, s, 28).mean((1, 3))
    m = mask.view(h, s, w, s).amax((1, 3)) > 0

    def grow(x, m, passes):
        for _ in range(passes):
            px = torch.nn.functional.pad(x * m[:, :, None], (0, 0, 1, 1, 1, 1))
            pm = torch.nn.functional.pad(m.double(), (1, 1, 1, 1))
            total, count = torch.zeros_like(x), torch.zeros_like(m, dtype=torch.float64)
            for dy in range(3):
                for dx in range(3):
                    if (dy, dx) != (1, 1):
                        total += px[dy:dy + h, dx:dx + w]
                        count += pm[dy:dy + h, dx:dx + w]
            new = ~m & (count > 0)
            x = torch.where(new[:, :, None], total / count.clamp(min=1)[:, :, None], x)
            m = m | new
        return x, m

    a, m = grow(x[:, :, :27].contiguous(), m, case["dilation"])
    b, _ = grow(x[:, :, 27:].contiguous(), m, case["dilation"])  # with the mask the first one grew
    return {"sh": a.reshape(-1), "env": b.reshape(-1), "mask": None}


def _rays_exact(case, seed):
    if _tris(case) * case["count"] > 2e10:
        return None
    sc = _scene(case, seed)
    V, N, UV = [], [], []
    for g in sc.geometries:
        i = np.asarray(g.indices).reshape(-1, 3)
        V.append(np.asarray(g.vertices)[i])
        N.append(np.asarray(g.normals)[i])
        UV.append(np.asarray(g.texture_uvs)[i])
    V, N, UV = (torch.from_numpy(np.concatenate(a)).to("cuda", torch.float64) for a in (V, N, UV))
    rays = _rays(case, seed).double()
    e1, e2 = V[:, 1] - V[:, 0], V[:, 2] - V[:, 0]
    n0 = torch.linalg.cross(e1, e2)
    out = {k: [] for k in ("position", "uv", "normal", "t")}
    step = max(1, 20_000_000 // len(V))
    for r in rays.split(step):
        o, d = r[:, None, 0:3], r[:, None, 3:6]
        # Moeller and Trumbore 1997, dot products with the pairs' common crosses
        det = -(r[:, 3:6] @ n0.T)
        s = o - V[None, :, 0]
        t = (s * n0[None]).sum(-1) / det
        c = torch.linalg.cross(s, d.expand_as(s))
        u = -(c * e2[None]).sum(-1) / -det
        v = (c * e1[None]).sum(-1) / -det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > r[:, 6:7]) & (t < r[:, 7:8])
        t = torch.where(ok, t, torch.full_like(t, float("inf")))
        best, k = t.min(1)
        hit = torch.isfinite(best)
        u, v = u.gather(1, k[:, None]), v.gather(1, k[:, None])
        b = torch.stack([1 - u - v, u, v], 1) * hit[:, None, None]
        nrm = (b * N[k]).sum(1)
        out["t"].append(torch.where(hit, best, torch.zeros_like(best)))
        out["position"].append(torch.where(hit[:, None], r[:, 0:3] + r[:, 3:6] * out["t"][-1][:, None],
                                           torch.zeros_like(nrm)))
        out["normal"].append(nrm / nrm.norm(dim=1, keepdim=True).clamp(min=1e-300))
        out["uv"].append((b * UV[k]).sum(1))
    return {**{k: torch.cat(v) for k, v in out.items()}, "material": None, "hit": None, "prim": None}


def exact(case, seed):
    if case["op"] == "post":
        return _post_exact(case, seed)
    if case["op"] == "rays":
        return _rays_exact(case, seed)
    if case["op"] in ("lightmap", "bake") and case["scene"] == "quad":
        return _quad_exact(case, seed)
    return None
