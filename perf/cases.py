"""The work that a program using this package has it do, as cases that can be timed and compared.

Each case goes through the package's public entry points at the sizes its configurations, tests and benchmark use:
whole clipmap frames (small room, 1M-triangle hall, a moving camera), the cone trace in its texture, FP16 and exact
forms, the sparse octree, a step of inverse fitting, a rendered camera frame and a batch of scenes.  ``exact``
restates the traced outputs (and the fit's gradients) in 64 bits with plain torch; rasterised outputs are bytes.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from vk_voxel_cone_tracing_gb300 import capi, clipmap, engine, fit, passes, render, scene

LIGHT = (0.3, -1.0, 0.2)
F64 = torch.float64


def listed():
    return [
        # the benchmark's configuration 1: a 34k-triangle room at R = 128, every level due (what a viewer pays on
        # load and on each cadence's first frame)
        dict(name="frame_room", kind="frame", scene="room", triangles=34000, R=128, shadow=2048, r8=False, index=0),
        # the headline frame: the 1M-triangle hall at R = 256
        dict(name="frame_hall", kind="frame", scene="hall", triangles=1000000, R=256, shadow=2048, r8=False, index=0),
        # a camera walking through a hall: two toroidal frames, one there and one back, on the radiance cadence
        dict(name="frame_walk", kind="walk", scene="hall", triangles=300000, R=128, shadow=2048, move=0.4),
        # the smallest trace of the batched configuration: launch count and latency
        dict(name="trace_small", kind="trace", scene="room", triangles=34000, R=64, samples=4096, fp16=False),
        # the headline trace: one sample per pixel of 1920x1080 on the hall's clipmap
        dict(name="trace_view", kind="trace", scene="hall", triangles=1000000, R=256, samples=2073600, fp16=False),
        # the FP16 storage form after a frame: conversion, FP16 mips, trace of an odd number of samples
        dict(name="trace_fp16", kind="trace", scene="hall", triangles=300000, R=128, samples=131071, fp16=True),
        # the exact FP32 drop-in on the linear atlas with configuration 1's 16 fixed 30-degree cones
        dict(name="trace_exact", kind="exact", scene="room", triangles=34000, R=128, samples=65536, degrees=30.0),
        # the octree method on configuration 1's room: fragment list, build (depth 7) and trace
        dict(name="svo_room", kind="svo", scene="room", triangles=34000, level=7, samples=65536, shadow=2048),
        # the large octree: displaced terrain and boxes at 512^3
        dict(name="svo_terrain", kind="svo", scene="terrain", triangles=4000000, level=9, samples=1000003, shadow=2048),
        # one Adam iteration of inverse radiance fitting (mips, trace, adjoint, mip adjoint, update)
        dict(name="fit_step", kind="fit", R=64, views=4, side=128),
        # a whole rendered frame, camera to image, as the command line runs it
        dict(name="render_hall", kind="render", scene="hall", triangles=300000, R=128, width=1280, height=720),
        # many small uneven scenes at once (the batched configuration, a part of its 64)
        dict(name="batch", kind="batch", scenes=16, low=10000, high=120000, most_samples=65536, streams=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "walk", "trace", "trace", "trace", "exact", "svo", "fit", "render", "batch"])
    room = rng.random() < 0.4
    triangles = _log(rng, 12000, 60000) if room else _log(rng, 20000, 800000)
    place = dict(scene="room" if room else "hall", triangles=triangles)
    if kind == "frame":
        return dict(kind=kind, **place, R=rng.choice([32, 64, 128, 128, 256]), shadow=rng.choice([512, 1000, 2048]),
                    r8=rng.random() < 0.4, index=rng.choice([0, 1, 2, 4, 16]))
    if kind == "walk":
        return dict(kind=kind, **place, R=rng.choice([64, 128, 256]), shadow=rng.choice([512, 2048]),
                    move=round(rng.uniform(0.05, 1.5), 3))
    if kind == "trace":
        R = rng.choice([64, 128, 128, 256])
        return dict(kind=kind, **place, R=R, samples=_log(rng, 1000, 1200000), fp16=rng.random() < 0.4)
    if kind == "exact":
        return dict(kind=kind, **place, R=rng.choice([32, 64, 128]), samples=_log(rng, 1000, 200000),
                    degrees=rng.choice([0.0, 0.0, 30.0, 40.0]))
    if kind == "svo":
        if rng.random() < 0.3:
            place = dict(scene="terrain", triangles=_log(rng, 150000, 1500000))
        return dict(kind=kind, **place, level=rng.choice([5, 6, 7, 8, 9]), samples=_log(rng, 1000, 500000),
                    shadow=rng.choice([512, 2048]))
    if kind == "fit":
        return dict(kind=kind, R=rng.choice([32, 64]), views=rng.choice([1, 2, 4]), side=rng.randrange(40, 150))
    if kind == "render":
        w = _log(rng, 160, 1920)
        return dict(kind=kind, **place, R=rng.choice([64, 128, 256]), width=w, height=w * 9 // 16)
    return dict(kind=kind, scenes=rng.randrange(4, 21), low=10000, high=rng.choice([40000, 120000]),
                most_samples=rng.choice([16384, 65536]), streams=rng.choice([2, 4]))


# ------------------------------------------------------------------ inputs

def _scene(name, triangles, seed):
    if name == "room":
        return scene.room_scene(seed, max(100, triangles - 14000))
    if name == "hall":
        return scene.hall_scene(seed, triangles)
    return scene.terrain_scene(seed, triangles, boxes=min(10000, triangles // 100))


def _camera(name):
    return {"room": (0.0, 4.0, 0.0), "hall": (0.0, 5.0, 0.0), "terrain": (0.0, 4.0, 0.0)}[name]


def _eye(name):
    return {"room": (1.0, 4.0, -4.0), "hall": (0.0, 5.0, -12.0), "terrain": (0.0, 8.0, -12.0)}[name]


def _light_shadow(camera):
    d = np.asarray(LIGHT, np.float64)
    d /= np.linalg.norm(d)
    return passes.light_shadow_desc(tuple((np.asarray(camera) - 15.0 * d).astype(np.float32).tolist()), LIGHT)


class State:
    """What a program keeps: scene, buffers, textures, descs (attributes set by the makers below)."""


def _frame_state(name, triangles, R, shadow, seed, r8=False, texture=True):
    s = State()
    s.scene = _scene(name, triangles, seed)
    s.ds, s.ws, s.R = passes.DeviceScene(s.scene), passes.Workspace(), R
    s.camera, s.eye = _camera(name), _eye(name)
    s.light, s.lsd = passes.light_desc(LIGHT), _light_shadow(s.camera)
    s.shadow = torch.empty((shadow, shadow), dtype=torch.float32, device="cuda")
    s.opacity = clipmap.new_atlas_r8(R) if r8 else clipmap.new_atlas(R)
    s.radiance = clipmap.new_atlas(R)
    s.tex = clipmap.RadianceTexture(R) if texture else None
    s.format = capi.OPACITY_R8 if r8 else capi.OPACITY_RGBA8
    s.state = (capi.ClipmapRegion * 6)()
    return s


def _frame(s, camera=None, index=0, revox=capi.REVOX_FULL):
    return passes.clipmap_frame(s.ds, camera or s.camera, s.R, s.opacity, s.radiance, s.shadow, s.light, s.lsd, s.ws,
                                frame_index=index, texture=s.tex, revoxelization=revox, regions_state=s.state,
                                opacity_format=s.format)


def _outputs(s, n):
    s.diffuse = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    s.specular = torch.zeros((n, 4), dtype=torch.float32, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        s = _frame_state(case["scene"], case["triangles"], case["R"], case["shadow"], seed, case["r8"])
        _frame(s)
        s.index = case["index"]
    elif kind == "walk":
        s = _frame_state(case["scene"], case["triangles"], case["R"], case["shadow"], seed)
        _frame(s)
        m = case["move"]
        s.there = (s.camera[0] + m, s.camera[1], s.camera[2] + 0.6 * m)
    elif kind in ("trace", "exact"):
        s = _frame_state(case["scene"], case["triangles"], case["R"], 2048, seed, texture=kind == "trace")
        s.regions = _frame(s)
        s.desc = clipmap.trace_desc(**scene.default_trace_desc(clipmap.regions_to_numpy(s.regions), s.R))
        n = case["samples"]
        s.samples = clipmap.samples_to_device(scene.surface_samples(s.scene, n, seed + 1))
        _outputs(s, n)
        s.aperture = math.radians(case.get("degrees", 0.0))
        if kind == "trace":
            s.scratch = clipmap.fast_scratch(n)
        if case.get("fp16"):
            s.tex16 = clipmap.RadianceTexture(s.R, capi.TEX_RGBA16F)
            s.atlas16 = clipmap.new_atlas_rgba16f(s.R)
            _fp16(s)
    elif kind == "svo":
        s = State()
        s.scene = _scene(case["scene"], case["triangles"], seed)
        s.ds, s.ws = passes.DeviceScene(s.scene), passes.Workspace()
        camera, s.eye = _camera(case["scene"]), _eye(case["scene"])
        s.light, s.lsd = passes.light_desc(LIGHT), _light_shadow(camera)
        s.shadow = torch.empty((case["shadow"],) * 2, dtype=torch.float32, device="cuda")
        passes.shadow_depth(s.ds, s.lsd, s.shadow, s.ws)
        s.level, R = case["level"], 1 << case["level"]
        s.desc = clipmap.trace_desc(**scene.default_trace_desc(clipmap.regions_to_numpy(clipmap.clip_regions(camera, R)), R))
        s.samples = clipmap.samples_to_device(scene.surface_samples(s.scene, case["samples"], seed + 1))
        # the list's and the pool's buffers, as a program keeps them from one frame to the next
        s.fragments = torch.zeros((400 * R * R + 1024, 2), dtype=torch.int32, device="cuda")
        s.pool = torch.zeros((1 << 23, 2), dtype=torch.int32, device="cuda")
    elif kind == "fit":
        s = _fit_state(case, seed)
    elif kind == "render":
        s = State()
        s.renderer = render.Renderer(_scene(case["scene"], case["triangles"], seed), R=case["R"], width=case["width"],
                                     height=case["height"])
        s.camera = _camera(case["scene"])
        s.renderer.render(s.camera, (0.6, -0.2, 0.77))
    else:
        s = _batch_state(case, seed)
    s.kind, s.fp16 = kind, bool(case.get("fp16"))
    return s


def _fp16(s):
    clipmap.to_rgba16f(s.radiance, s.R, out=s.atlas16, mirror=s.tex16)
    clipmap.cmd_downsample_rgba16f_all(s.atlas16, s.R, s.regions, 1, mirror=s.tex16)


def _fit_state(case, seed):
    s = State()
    R, n = case["R"], case["views"] * case["side"] ** 2
    regions = clipmap.clip_regions((0.0, 0.0, 0.0), R)
    s.regions = clipmap.regions_to_numpy(regions)
    s.desc = clipmap.trace_desc(**scene.default_trace_desc(s.regions, R))
    s.samples = clipmap.samples_to_device(scene.random_samples(n, (0, 0, 0), 5.0, seed=seed, specular_fraction=1.0))
    s.eye = (0.0, 1.0, -4.0)
    s.light = passes.light_desc(LIGHT)
    s.init = scene.smooth_volume(R, seed + 1, xp=torch, device="cuda").reshape(-1).contiguous()
    s.fit = fit.RadianceFit(R, regions, s.desc, clipmap.cam_matrix(s.eye), s.light, s.samples, lr=0.005, init=s.init)
    hidden = scene.smooth_volume(R, seed + 2, xp=torch, device="cuda").reshape(-1).contiguous()
    s.target = s.fit.render(hidden)
    s.fit.set_targets(*s.target)
    return s


def _batch_state(case, seed):
    s = State()
    rng = np.random.default_rng(case["scenes"])  # the sizes are the case's, the scenes the seed's
    grids = rng.choice([64, 64, 128], size=case["scenes"])
    contexts = {int(R): [engine.Context(int(R), 1024) for _ in range(4)] for R in sorted(set(grids.tolist()))}
    s.jobs, s.keep, s.outs, s.streams, dealt = [], [], [], case["streams"], {}
    light = passes.light_desc(LIGHT)
    for k, R in enumerate(grids.tolist()):
        T = int(math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"]))))
        n = int(math.exp(rng.uniform(math.log(4096), math.log(case["most_samples"]))))
        sc = scene.hall_scene(seed + k, T)
        ds = passes.DeviceScene(sc)
        samples = clipmap.samples_to_device(scene.surface_samples(sc, n, seed + k))
        d = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        sp = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        camera = _camera("hall")
        desc = clipmap.trace_desc(**scene.default_trace_desc(clipmap.regions_to_numpy(clipmap.clip_regions(camera, R)), R))
        ctx = contexts[R][dealt.get(R, 0) % 4]
        dealt[R] = dealt.get(R, 0) + 1
        s.jobs.append(engine.batch_job(ctx, ds, camera, light, _light_shadow(camera), desc, _eye("hall"), samples, d, sp))
        s.keep.append((ctx, ds, samples))
        s.outs += [d, sp]
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    if s.kind == "frame":
        _frame(s, index=s.index)
        return [s.opacity, s.radiance, s.shadow]
    if s.kind == "walk":
        _frame(s, s.there, 1, capi.REVOX_TOROIDAL)
        _frame(s, s.camera, 2, capi.REVOX_TOROIDAL)
        return [s.opacity, s.radiance, s.shadow]
    if s.kind == "trace":
        if s.fp16:
            _fp16(s)
        clipmap.cone_trace_fast(s.desc, s.eye, s.tex16 if s.fp16 else s.tex, s.samples, light=s.light, shadow=s.shadow,
                                shadow_desc=s.lsd, diffuse=s.diffuse, specular=s.specular, scratch=s.scratch)
        return [s.diffuse, s.specular] + ([s.atlas16.view(torch.float16)] if s.fp16 else [])
    if s.kind == "exact":
        clipmap.cone_trace(s.desc, s.eye, s.radiance, s.R, s.samples, light=s.light, shadow=s.shadow, shadow_desc=s.lsd,
                           diffuse=s.diffuse, specular=s.specular, diffuse_aperture=s.aperture)
        return [s.diffuse, s.specular]
    if s.kind == "svo":
        f = passes.svo_fragments(s.ds, s.level, s.shadow, s.light, s.lsd, s.ws, out=s.fragments)
        nodes = C.c_int64(0)
        capi.call("vct_svo_build", C.c_void_p(f.data_ptr()), f.shape[0], s.level, C.c_void_p(s.pool.data_ptr()),
                  s.pool.shape[0], capi.SVO_DETERMINISTIC, C.byref(nodes), s.ws.handle,
                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
        d, sp = passes.svo_cone_trace(s.desc, s.eye, s.pool, nodes.value, s.samples, bb_min=s.ds.bb_min,
                                      bb_max=s.ds.bb_max, light=s.light, shadow=s.shadow, shadow_desc=s.lsd)
        return {"fragments": s.fragments, "pool": s.pool, "nodes": nodes.value, "diffuse": d, "specular": sp}
    if s.kind == "fit":
        loss = s.fit.step()
        return {"loss": loss, "diffuse": s.fit.dout, "specular": s.fit.sout, "param": s.fit.param, "m": s.fit.m,
                "v": s.fit.v}
    if s.kind == "render":
        return s.renderer.render(s.camera, (0.6, -0.2, 0.77))
    engine.batch_submit(s.jobs, s.streams)
    return s.outs


# Cone samples per surface sample of the default cones in these scenes (the benchmark counts 349 on the hall at
# R = 256), and the arithmetic of one: six trilinear fetches of four channels, their weights and the composite.
_STEPS, _FLOPS = 350, 400


def work(case):
    kind, T = case["kind"], case.get("triangles", 0)
    if kind in ("frame", "walk"):
        R = case["R"]
        levels = 6 if kind == "walk" else sum(case["index"] % (1 << l) == 0 for l in range(6))
        texels = 6 * R ** 3
        opacity = 6 * texels * (1 if case.get("r8") else 4)
        # geometry once; the opacity written, the due radiance levels written to the atlas and the texture; the map
        return {"bytes": 84 * T + opacity + 2 * 4 * texels * levels + 4 * case["shadow"] ** 2, "flops": 6 * 100.0 * T}
    if kind in ("trace", "exact"):
        n, texels = case["samples"], 36 * case["R"] ** 3
        extra = texels * 12 if case.get("fp16") else 0
        return {"bytes": 112 * n + extra, "flops": float(n) * _STEPS * _FLOPS}
    if kind == "svo":
        n = case["samples"]
        # geometry, one 8-byte fragment per covered sample (these scenes have 50 to 220 a texel of the grid's face), the trace
        fragments = 150.0 * 4 ** case["level"]
        return {"bytes": 84.0 * T + 16 * fragments + 112 * n, "flops": float(n) * 190 * 60}
    if kind == "fit":
        n = case["views"] * case["side"] ** 2
        floats = 4 * 36 * case["R"] ** 3
        return {"bytes": 112.0 * n + 4 * floats * 7, "flops": float(n) * _STEPS * _FLOPS * 3}
    if kind == "render":
        n, R = case["width"] * case["height"], case["R"]
        return {"bytes": 84 * T + 36 * R ** 3 * 12 + 4 * 2048 ** 2 + 250 * n, "flops": float(n) * 90 * _FLOPS}
    mean = math.sqrt(4096 * case["most_samples"])
    return {"bytes": case["scenes"] * (36 * 80 ** 3 * 12 + 84 * case["low"] + 112 * mean),
            "flops": case["scenes"] * mean * _STEPS * _FLOPS}


# ------------------------------------------------------------------ in 64 bits

_DIRS = [(0.57735, 0.57735, 0.57735), (0.57735, -0.57735, -0.57735), (-0.57735, 0.57735, -0.57735),
         (-0.57735, -0.57735, 0.57735), (-0.903007, -0.182696, -0.388844), (-0.903007, 0.182696, 0.388844),
         (0.903007, -0.182696, 0.388844), (0.903007, 0.182696, -0.388844), (-0.388844, -0.903007, -0.182696),
         (0.388844, -0.903007, 0.182696), (0.388844, 0.903007, -0.182696), (-0.388844, 0.903007, 0.182696),
         (-0.182696, -0.388844, -0.903007), (0.182696, 0.388844, -0.903007), (-0.182696, 0.388844, 0.903007),
         (0.182696, -0.388844, 0.903007)]


def _f64(x):
    return torch.tensor([float(v) for v in x], dtype=F64, device="cuda")


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


class Clip64:
    """Trilinear samples of a clipmap's texel table ((texels, 4), any type) at integer levels."""

    def __init__(self, texels, scale, R, voxel):
        self.t, self.scale, self.R, self.voxel = texels, scale, R, voxel

    def __call__(self, p, level, dirs):
        R, rb = self.R, self.R + 2
        W = 6 * rb
        ext = self.voxel * torch.exp2(level.to(F64)) * R
        q = p / ext[:, None]
        q = (q - q.floor()) * R + 0.5
        base = q.floor()
        fr, base = q - base, base.long()
        out = 0.0
        for a in range(3):
            face = torch.where(dirs[:, a] > 0, 2 * a, 2 * a + 1)
            x0, y0 = base[:, 0] + face * rb, base[:, 1] + level * rb
            tap = 0.0
            for k in range(8):
                dx, dy, dz = k & 1, (k >> 1) & 1, k >> 2
                w = ((fr[:, 0] if dx else 1 - fr[:, 0]) * (fr[:, 1] if dy else 1 - fr[:, 1]) *
                     (fr[:, 2] if dz else 1 - fr[:, 2]))
                i = ((base[:, 2] + dz) * W + y0 + dy) * W + x0 + dx
                tap = tap + self.t.index_select(0, i).to(F64) * w[:, None]
            out = out + tap * (dirs[:, a] ** 2)[:, None]
        return out * self.scale


class Octree64:
    """Point samples of a node pool at resolution 2^level."""

    def __init__(self, pool, lo, hi, dim):
        self.child = (pool[:, 0] & 0x7fffffff).long()
        self.rgba = pool.view(torch.uint8).reshape(-1, 8)[:, 4:]
        self.c, self.ev, self.dim = (lo + hi) / 2, (hi - lo).max() / 2, dim

    def __call__(self, p, level, dirs):
        u = ((p - self.c) / self.ev + 1) / 2 * self.dim
        f = u.clamp(0, self.dim).long()
        res, target = self.dim, 1 << level
        cur, idx = torch.zeros_like(level), torch.zeros_like(level)
        going = torch.ones_like(level, dtype=torch.bool)
        while res > 1:
            res //= 2
            b = (f >= res).long()
            idx = torch.where(going, cur + (b[:, 2] | (b[:, 0] << 1) | (b[:, 1] << 2)), idx)
            cur = torch.where(going, self.child[idx], cur)
            f = f - b * res
            going = going & (cur != 0) & (target < res)
        return self.rgba[idx].to(F64) / 255


def _march(fetch, d, start, dirs, coef, start_level, factor):
    """traceCone for every row, rows dropped as they end: (rgb, 1 - occlusion)."""
    n = start.shape[0]
    uvs = d.voxel_size
    start = start + dirs * (uvs * torch.exp2(start_level) * d.trace_start_offset * 0.5)[:, None]
    center, radius = _f64(d.volume_center), uvs * d.volume_dimension / 2
    out_rgb, out_occ = torch.zeros((n, 3), dtype=F64, device="cuda"), torch.zeros(n, dtype=F64, device="cuda")
    done_rows, done_rgb, done_occ = [], [], []
    rows = torch.arange(n, device="cuda")
    step = torch.zeros(n, dtype=F64, device="cuda")
    diameter = torch.full_like(step, uvs)
    seg = uvs * torch.exp2(start_level)
    rgb, alpha, occ = out_rgb, out_occ, out_occ
    while rows.numel():
        pos = start + dirs * step[:, None]
        with torch.no_grad():
            dist = (center - pos).norm(dim=1)
            cur = torch.maximum(torch.maximum(start_level, torch.log2(diameter / uvs)), torch.log2(dist / radius).ceil())
            cur = cur.clamp(max=5.0)
            low = cur.floor()
            fr = (cur - low)[:, None]
        s = fetch(pos, low.long(), dirs) * (1 - fr) + fetch(pos, cur.ceil().long(), dirs) * fr
        vs = uvs * torch.exp2(cur)
        corr = seg / vs
        opacity = (1 - (1 - s[:, 3]).clamp(min=0) ** corr).clamp(0, 1)
        k = (1 - alpha).clamp(0, 1)
        rgb = rgb + (k * corr)[:, None] * s[:, :3]
        alpha = alpha + k * opacity
        occ = occ + (1 - occ) * opacity / (1 + (step + vs) * d.occlusion_decay)
        new = step + diameter.clamp(min=uvs) * factor
        seg, step = new - step, new
        diameter = step * coef
        go = (step < 30.0) & (occ < 1.0)
        if not bool(go.all()):
            end = (~go).nonzero()[:, 0]
            done_rows.append(rows[end]), done_rgb.append(rgb[end]), done_occ.append(occ[end])
            keep = go.nonzero()[:, 0]
            rows, start, dirs, coef, start_level = rows[keep], start[keep], dirs[keep], coef[keep], start_level[keep]
            step, seg, diameter, rgb, alpha, occ = (x[keep] for x in (step, seg, diameter, rgb, alpha, occ))
    if not done_rows:
        return torch.zeros((0, 4), dtype=F64, device="cuda")
    at = torch.argsort(torch.cat(done_rows))
    return torch.cat([torch.cat(done_rgb)[at], 1 - torch.cat(done_occ)[at][:, None]], 1)


def _visibility(shadow, lsd, wp):
    if shadow is None:
        return 1.0
    H, W = shadow.shape
    V, P = _f64(lsd.view).reshape(4, 4).T, _f64(lsd.proj).reshape(4, 4).T
    l = wp @ V[:2, :3].T + V[:2, 3]
    c = (l @ P[:2, :2].T + P[:2, 3]) * 0.5 + 0.5
    padded = torch.nn.functional.pad(shadow.to(F64), (1, 1, 1, 1))
    total = 0.0
    for yi in range(4):
        for xi in range(4):
            u, v = c[:, 0] * W + (xi - 1.5) - 0.5, c[:, 1] * H + (yi - 1.5) - 0.5
            i, j = u.floor(), v.floor()
            a, b = u - i, v - j
            at = lambda dx, dy: padded[(j + dy + 1).clamp(0, H + 1).long(), (i + dx + 1).clamp(0, W + 1).long()]
            total = total + (at(0, 0) * (1 - a) + at(1, 0) * a) * (1 - b) + (at(0, 1) * (1 - a) + at(1, 1) * a) * b
    return (total / 16)[:, None]


def _direct(wp, normal, view, dcol, scol, rough, emission, light, shadow, lsd):
    l = _unit(-_f64(light.direction))
    h = _unit(l + view)
    dot = lambda a, b: (a * b).sum(1)
    nl, nv = dot(normal, l.expand_as(normal)).clamp(0.001, 1), dot(normal, view).abs().clamp(0.001, 1)
    nh, vh = dot(normal, h).clamp(0, 1), dot(view, h).clamp(0, 1)
    ar = rough * rough
    r90 = (scol.max(1).values * 50).clamp(0, 1)[:, None]
    F = scol + (r90 - scol) * ((1 - vh).clamp(0, 1) ** 5)[:, None]
    att = lambda x: 2 * x / (x + (ar * ar + (1 - ar * ar) * x * x).sqrt())
    rs = ar * ar
    f = (nh * rs - nh) * nh + 1
    D = rs / (3.141592 * f * f)
    c = nl[:, None] * ((1 - F) * dcol / 3.141592 + F * (att(nl) * att(nv) * D / (4 * nl * nv))[:, None])
    c = c * _visibility(shadow, lsd, wp)
    return torch.where((emission > 0).any(1, keepdim=True), emission, c)


def _trace64(fetch, d, eye, samples, light, shadow, lsd, aperture=0.872665, octree=False):
    """The GI output mode: (diffuse, specular) of every sample."""
    g = samples.to(F64)
    wp, dcol, rough = g[:, 0:3], g[:, 8:11], g[:, 11]
    scol, metal, emission = g[:, 12:15], g[:, 15], g[:, 16:19]
    view, normal = _unit(_f64(eye) - wp), _unit(g[:, 4:7] * 2 - 1)
    uvs, n = d.voxel_size, g.shape[0]
    dist, radius = (_f64(d.volume_center) - wp).norm(dim=1), d.voxel_size * d.volume_dimension / 2
    up = torch.log2(dist / radius).clamp(min=0).ceil()
    f = dist / (radius * torch.exp2(up))
    level = torch.where(f > 0.5, up + (f - 0.5) * 2, up)
    start = wp + normal * (uvs * torch.exp2(level) * d.trace_start_offset)[:, None]
    factor = max(0.2, d.min_trace_step_factor)
    total = torch.zeros((n, 4), dtype=F64, device="cuda")
    total[:, 3] = 1.0
    weight = torch.zeros(n, dtype=F64, device="cuda")
    coef = 2 * math.tan(aperture / 2)
    for c in range(16):
        dirs = torch.tensor(_DIRS[c], dtype=F64, device="cuda").expand(n, 3)
        cos = (normal * dirs).sum(1)
        at = (cos >= 0).nonzero()[:, 0]
        for i in at.split(1 << 20):
            r = _march(fetch, d, start[i], dirs[i], torch.full_like(level[i], coef), level[i], factor)
            r = r.clamp(0, 1) if octree else r
            total = total.index_add(0, i, r * cos[i][:, None])
        weight = weight.index_add(0, at, cos[at])
    ind = total / weight[:, None] if octree else total / 16
    ao = ind[:, 3:] * d.ambient_occlusion_factor
    rgb = ind[:, :3] * dcol * d.indirect_diffuse_intensity
    direct = _direct(wp, normal, view, dcol, scol, rough, emission, light, shadow, lsd)
    if octree:
        ao, rgb, direct = ao.clamp(0, 1), rgb.clamp(0, 1), direct.clamp(0, 1)
    spec = torch.zeros((n, 3), dtype=F64, device="cuda")
    at = ((scol > 1e-6).any(1) & (metal > 1e-6)).nonzero()[:, 0]
    refl = -view + normal * (2 * (normal * view).sum(1, keepdim=True))
    refl = _unit(refl) if octree else refl
    for i in at.split(1 << 18):
        ap = 2 * torch.tan(rough[i].clamp(min=0.05) / 2)
        r = _march(fetch, d, start[i], refl[i], ap, level[i], max(0.2, uvs) if octree else uvs)
        r = r.clamp(0, 1) if octree else r
        spec = spec.index_add(0, i, r[:, :3] * scol[i] * d.indirect_specular_intensity)
    one = torch.ones((n, 1), dtype=F64, device="cuda")
    return torch.cat([direct * ao + rgb, one], 1), torch.cat([spec, one], 1)


def _mips64(vol, regions, R):
    """Radiance mips of levels 1..5 of a (texels, 4) float clipmap."""
    rb, half = R + 2, R // 2
    v = vol.reshape(rb, 6, rb, 6, rb, 4)
    levels = [v[:, l] for l in range(6)]
    for l in range(1, 6):
        cur = [torch.tensor([int(regions[l - 1, a]) // 2 + i for i in range(half)], device="cuda") for a in range(3)]
        lerp = []
        for a in range(3):
            c = (int(regions[l - 1, a]) >> 1) + (half >> 1)
            lerp.append((cur[a] + 0.5 - c).abs() - 0.5)
        far = torch.maximum(torch.maximum(lerp[0][None, None, :], lerp[1][None, :, None]), lerp[2][:, None, None])
        edge = (half >> 1) - capi.DOWNSAMPLE_REGION_SIZE
        lerp = torch.where(far >= edge, (far - edge + 1) / (capi.DOWNSAMPLE_REGION_SIZE + 1), 0.0).to(F64)[..., None]
        w = [(c % R) + 1 for c in cur]
        p = [((2 * c) % R) + 1 for c in cur]
        prev, faces = levels[l - 1], []
        child = lambda x, a, b: x.index_select(a, p[2 - a] + b)
        for f in range(6):
            block = prev[:, :, f]  # z, y, x, c
            total = 0.0
            axis = f >> 1  # 0 x, 1 y, 2 z
            others = [a for a in range(3) if a != axis]
            for k in range(4):
                bits = {others[0]: k & 1, others[1]: k >> 1}
                pair = []
                for j in range(2):
                    bits[axis] = j ^ (f & 1)
                    pair.append(child(child(child(block, 0, bits[2]), 1, bits[1]), 2, bits[0]))
                total = total + pair[0] + (1 - pair[0][..., 3:]) * pair[1]
            own = levels[l][:, :, f].index_select(0, w[2]).index_select(1, w[1]).index_select(2, w[0])
            new = levels[l][:, :, f].clone()
            new[w[2][:, None, None], w[1][None, :, None], w[0][None, None, :]] = total / 4 * (1 - lerp) + own * lerp
            faces.append(new)
        levels[l] = torch.stack(faces, 2)
    return torch.stack(levels, 1).reshape(-1, 4)


def _fit64(s, R):
    vol = s.init.to(F64).reshape(-1, 4).requires_grad_(True)
    work = _mips64(vol, s.regions, R)
    leaf = work.detach().requires_grad_(True)
    n = s.samples.shape[0]
    loss, outs = 0.0, []
    for i in torch.arange(n, device="cuda").split(8192):
        out = _trace64(Clip64(leaf, 1.0, R, s.desc.voxel_size), s.desc, s.eye, s.samples[i], s.light, None, None)
        part = sum(((o - t[i].to(F64)) ** 2).sum() for o, t in zip(out, s.target)) / (8 * n)
        part.backward()
        loss += float(part)
        outs.append([o.detach() for o in out])
    work.backward(leaf.grad)
    g = vol.grad
    b1, b2 = s.fit.adam.beta1, s.fit.adam.beta2
    m, v = (1 - b1) * g, (1 - b2) * g * g
    p = vol.detach() - s.fit.adam.lr * g / (g.abs() + s.fit.adam.eps)
    p = torch.cat([p[:, :3].clamp(min=0), p[:, 3:].clamp(0, s.fit.adam.alpha_hi)], 1)
    d, sp = (torch.cat(o) for o in zip(*outs))
    return {"loss": loss, "diffuse": d, "specular": sp, "param": p.reshape(-1), "m": m.reshape(-1), "v": v.reshape(-1)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("trace", "exact"):
        if case["samples"] > 140000:
            return None
        s = prepare(case, seed)
        voxel = s.desc.voxel_size
        if case.get("fp16"):
            fetch = Clip64(s.atlas16.view(torch.float16).reshape(-1, 4), 1.0, s.R, voxel)
        else:
            fetch = Clip64(s.radiance.view(torch.uint8).reshape(-1, 4), 1 / 255, s.R, voxel)
        aperture = math.radians(case["degrees"]) if case.get("degrees") else 0.872665
        out = list(_trace64(fetch, s.desc, s.eye, s.samples, s.light, s.shadow, s.lsd, aperture))
        return out + ([None] if case.get("fp16") else [])
    if kind == "svo":
        if case["samples"] > 1100000:
            return None
        s = prepare(case, seed)
        r = run(s)  # the fragment list and the pool are whole numbers: only the trace is restated
        lo, hi = (torch.from_numpy(b).to("cuda", F64) for b in (s.ds.bb_min, s.ds.bb_max))
        d, sp = _trace64(Octree64(r["pool"], lo, hi, 1 << case["level"]), s.desc, s.eye, s.samples, s.light, s.shadow,
                         s.lsd, octree=True)
        return {"fragments": None, "pool": None, "nodes": None, "diffuse": d, "specular": sp}
    if kind == "fit":
        return _fit64(prepare(case, seed), case["R"])
    return None
