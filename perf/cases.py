"""The renderer's performance cases: what a program that uses the library asks of it, from a
thumbnail to the headline frame, each through the public entry points of ``merian_gb300``.

A case's scene is resident before the call, as in a renderer that shows one scene for many frames
(scenes are kept by what describes them); what changes from pass to pass is what changes from frame
to frame: the camera, the random sequence ("frame"), the pixel list or the rays. Sizes are those
of the package's own workloads (``merian_gb300/scene.py``, ``workloads.py``) and odd ones between
them.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from merian_gb300 import _native as N
from merian_gb300 import node
from merian_gb300 import scene as S
from merian_gb300 import workloads as W


def listed():
    return [
        # a thumbnail of a small room: the smallest request, where launches and latency count
        dict(name="thumbnail-64", op="render", scene="cornell", triangles=1024, width=64, height=64,
             spp=1, length=5, nee=True, rr=3, sort=False, demodulate=False, pixels=0),
        # the reference's own estimator on its strict-parity configuration
        dict(name="room-256-16spp", op="render", scene="cornell", triangles=1024, width=256,
             height=256, spp=16, length=5, nee=False, rr=0, sort=False, demodulate=False, pixels=0),
        # a list of pixels to refine (adaptive sampling, network tiles), material-sorted shading,
        # BSDF sampling only, result on the host
        dict(name="pixels-37003", op="render", scene="soup", triangles=200_000, width=1920,
             height=1080, spp=8, length=8, nee=False, rr=0, sort=True, demodulate=False,
             pixels=37_003),
        # an ordinary preview frame of a large scene
        dict(name="soup-360p-16spp", op="render", scene="soup", triangles=1_000_000, width=640,
             height=360, spp=16, length=8, nee=True, rr=3, sort=False, demodulate=False, pixels=0),
        # the benchmark frame, material-sorted as the benchmark's tuning has it: the largest
        dict(name="soup-1080p-64spp", op="render", scene="soup", triangles=1_000_000, width=1920,
             height=1080, spp=64, length=8, nee=True, rr=3, sort=True, demodulate=False, pixels=0),
        # an instanced, textured scene with long paths
        dict(name="instanced-720p-4spp", op="render", scene="instanced", triangles=400_000,
             width=1280, height=720, spp=4, length=16, nee=True, rr=3, sort=False,
             demodulate=False, pixels=0),
        # many small requests over many scenes in one call
        dict(name="batch-48", op="batch", requests=48, scenes=12, largest=300_000),
        # the request server under a burst of small requests
        dict(name="served-32", op="serve", requests=32, scenes=12, largest=300_000),
        # the visibility and material buffer of a frame
        dict(name="gbuffer-1080p", op="gbuffer", scene="instanced", triangles=400_000, width=1920,
             height=1080),
        # the caller's own rays, incoherent: closest hits in the large scene
        dict(name="rays-closest-1m", op="rays", scene="soup", triangles=1_000_000,
             rays=1_000_003, any=False),
        # ... and occlusion (ambient visibility) in a tessellated room
        dict(name="rays-occlusion-250k", op="rays", scene="cornell", triangles=102_400,
             rays=250_007, any=True),
        # an interactive viewer: G-buffer, one sample per pixel, accumulation; shown after 8 frames
        dict(name="progressive-540p", op="progressive", scene="soup", triangles=200_000, width=960,
             height=540, iterations=8, length=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng):
    kind = rng.choice(["cornell", "soup", "soup", "instanced"])
    if kind == "cornell":
        return dict(scene=kind, triangles=1024 * _log(rng, 1, 10) ** 2)
    if kind == "soup":
        return dict(scene=kind, triangles=_log(rng, 2_000, 1_000_000))
    return dict(scene=kind, triangles=100_000 * rng.randint(1, 4))


def draw(rng: random.Random):
    op = rng.choice(["render"] * 6 + ["batch", "serve", "gbuffer", "rays", "rays", "progressive"])
    if op == "batch" or op == "serve":
        return dict(op=op, requests=_log(rng, 3, 64), scenes=rng.randint(2, 12),
                    largest=_log(rng, 20_000, 300_000))
    c = dict(op=op, **_draw_scene(rng))
    if op == "rays":
        c.update(rays=_log(rng, 100, 1_000_000), any=rng.random() < 0.5)
        return c
    width = _log(rng, 33, 1920)
    height = max(17, int(width / rng.choice([1.0, 1.0, 4 / 3, 16 / 9, 2.1])))
    c.update(width=width, height=min(height, 1080))
    if op == "progressive":
        c.update(iterations=rng.randint(1, 12), length=rng.randint(3, 8))
    elif op == "render":
        # at most about a quarter of the benchmark frame's samples (small scenes have longer
        # paths: the box is nearly closed)
        spp = min(_log(rng, 1, 64), max(1, 32_000_000 // (c["width"] * c["height"])))
        nee = rng.random() < 0.6
        pixels = 0
        if rng.random() < 0.2:
            pixels = _log(rng, 50, max(51, c["width"] * c["height"] // 2))
        c.update(spp=spp, length=rng.choice([2, 5, 5, 8, 8, 16]), nee=nee, rr=3 if nee else 0,
                 sort=rng.random() < 0.3, demodulate=rng.random() < 0.2, pixels=pixels)
    return c


# ---- what the program keeps: a context on a stream of its own, and its scenes -------------------
class _Program:
    def __init__(self):
        self.stream = torch.cuda.Stream()
        self.ctx = S.Context(0, stream=self.stream.cuda_stream)
        self.scenes = {}
        self.serving = False

    def scene(self, kind: str, triangles: int):
        """(scene id, triangles that can be seen, environment texels)"""
        key = (kind, triangles)
        if key not in self.scenes:
            if kind == "cornell":
                data = S.cornell(tess=max(1, round(math.sqrt(triangles / 1024))))
            elif kind == "soup":
                # the 512x256 environment of the request mixes; the benchmark's 2048x1024 one for
                # its million triangles
                env = (2048, 1024) if triangles >= 1_000_000 else (512, 256)
                data = S.soup(n_triangles=triangles,
                              n_geometries=4096 if triangles >= 1_000_000 else
                              max(1, min(4096, triangles // 64)), env_size=env)
            else:
                data = W.instanced_scene(n_meshes=max(1, triangles // 50_000), n_instances=400,
                                         n_textures=32, tex_size=256)
            self.scenes[key] = self.ctx.upload(data)
        return self.scenes[key]

    def serve(self):
        if not self.serving:
            self.ctx.server_start(arena_bytes=1 << 30)
            self.serving = True


_program = None


def _get():
    global _program
    if _program is None:
        _program = _Program()
    return _program


def _camera(kind, width, height, rng):
    """The scene's camera, moved a little: the next frame of a walk through it."""
    d = [rng.uniform(-0.05, 0.05) for _ in range(3)]
    if kind == "cornell":
        pos, target, fov = (0.5, 0.5, -1.4), (0.5, 0.5, 0.0), 40.0
    elif kind == "soup":
        pos, target, fov = (0.5, 0.5, -0.6), (0.5, 0.5, 0.5), 45.0
    else:
        pos, target, fov = (50.0, 50.0, -45.0), (50.0, 50.0, 50.0), 60.0
        d = [100.0 * x for x in d]
    pos = tuple(p + x for p, x in zip(pos, d))
    return S.look_at(pos, target, (0.0, 1.0, 0.0), fov, width / height)


def _pool(case):
    """The scenes of the request mixes: (kind, triangles), sizes spread up to the largest."""
    n, hi = case["scenes"], case["largest"]
    out = []
    for i in range(n):
        t = round(math.exp(math.log(1024) + (math.log(hi) - math.log(1024)) * i / max(1, n - 1)))
        if i % 2:
            out.append(("soup", t))
        else:
            out.append(("cornell", 1024 * max(1, round(math.sqrt(min(t, 102_400) / 1024))) ** 2))
    return out


def _mix(case):
    """The requests of a case: (scene index, size, spp), the same for every seed."""
    rng = random.Random(case["requests"] * 1009 + case["scenes"])
    out = []
    for _ in range(case["requests"]):
        w, h = rng.choice(W.SMALL_RESOLUTIONS)
        out.append((rng.randrange(case["scenes"]), w, h, rng.choice(W.SMALL_SPP)))
    return out


def _rays(case, seed):
    """Incoherent rays: origins and directions uniform, as a caller's own bounces or probes."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["rays"]
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    side = 100.0 if case["scene"] == "instanced" else 1.0
    o = torch.rand((n, 3), generator=g, device="cuda")
    if case["scene"] == "cornell":
        o = 0.02 + 0.96 * o  # inside the room
    d = torch.randn((n, 3), generator=g, device="cuda")
    rays[:, 0:3] = o * side
    rays[:, 3] = 0.0
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    # occlusion within a radius, closest hits to the far plane
    rays[:, 7] = 0.25 * side if case["any"] else 1000.0
    return rays


def prepare(case, seed):
    p = _get()
    rng = random.Random(seed)
    op = case["op"]
    s = dict(op=op, p=p)
    if op in ("batch", "serve"):
        pool = _pool(case)
        ids = [p.scene(*k) for k in pool]
        jobs = []
        for k, (i, w, h, spp) in enumerate(_mix(case)):
            kind = pool[i][0]
            prm, _ = S.render_params(w, h, spp, 5 if kind == "cornell" else 8, nee=True,
                                     rr_depth=3, frame=(seed + k) % (1 << 30))
            jobs.append((ids[i], _camera(kind, w, h, rng), prm))
        s["jobs"] = jobs
        if op == "serve":
            p.serve()
            s["out"] = [np.zeros((j[2].width * j[2].height, 4), np.float32) for j in jobs]
        return s
    s["sid"] = p.scene(case["scene"], case["triangles"])
    if op == "rays":
        s["rays"] = _rays(case, seed)
        s["hits"] = torch.zeros((case["rays"], 8), dtype=torch.int32, device="cuda")
        s["any"] = case["any"]
        return s
    w, h = case["width"], case["height"]
    s["size"] = (w, h)
    s["cam"] = _camera(case["scene"], w, h, rng)
    if op == "gbuffer":
        s["out"] = torch.zeros((h * w, 16), dtype=torch.int32, device="cuda")
    elif op == "progressive":
        s["iterations"] = case["iterations"]
        s["graph"] = node.Graph(p.ctx, {"nodes": {
            "gbuffer": {"type": "GBuffer (Raytraced)", "properties": {"width": w, "height": h},
                        "outputs": ["gbuffer->render.gbuffer"]},
            "render": {"type": "Render (Path-traced)", "outputs": ["irradiance->accumulate.src"],
                       "properties": {"samples per pixel": 1, "max path length": case["length"],
                                      "next event estimation": True, "russian roulette depth": 3,
                                      "seed": seed % (1 << 30)}},
            "accumulate": {"type": "Accumulate",
                           "properties": {"alpha": 1.0, "inf history": True}}}})
    else:
        pix = None
        if case["pixels"]:
            pix = np.sort(np.random.default_rng(seed).choice(w * h, case["pixels"], replace=False))
        s["prm"], s["keep"] = S.render_params(
            w, h, case["spp"], case["length"], nee=case["nee"], rr_depth=case["rr"],
            sort_materials=case["sort"], demodulate_albedo=case["demodulate"],
            frame=seed % (1 << 30), pixels=pix)
        if pix is None:
            s["out"] = torch.zeros((h * w, 4), dtype=torch.float32, device="cuda")
    return s


def run(s):
    ctx, op = s["p"].ctx, s["op"]
    if op == "render":
        if s["keep"] is not None:  # a pixel list: to the host
            return ctx.render(s["sid"], s["cam"], s["prm"])
        ctx.render_device(s["sid"], s["cam"], s["prm"], s["out"].data_ptr())
        return s["out"]
    if op == "batch":
        return ctx.render_batch(s["jobs"])
    if op == "serve":
        tickets = [ctx.submit(sid, cam, prm, out_host=out)
                   for (sid, cam, prm), out in zip(s["jobs"], s["out"])]
        for t in tickets:
            rc, st = ctx.wait(t)
            N.check(rc)
            ctx.release(t)
        return s["out"]
    if op == "rays":
        n = s["rays"].shape[0]
        ctx.trace(s["sid"], s["rays"].data_ptr(), n, s["hits"].data_ptr(), any_hit=s["any"])
        t = s["hits"].view(torch.float32)[:, 6]
        if s["any"]:  # what an occlusion query says: blocked or not
            with torch.cuda.stream(s["p"].stream):
                return t >= 0.0
        return {"ids": s["hits"][:, 0:4], "barycentrics": s["hits"].view(torch.float32)[:, 4:6],
                "t": t}
    if op == "gbuffer":
        w, h = s["size"]
        N.check(ctx.lib.gbpt_gbuffer(ctx.handle, s["sid"], C.byref(s["cam"]), w, h, 0xFF,
                                     s["out"].data_ptr()))
        f = s["out"].view(torch.float32)
        # encoded normal, ids, half-precision pairs as bits; depth, albedo and emission
        return {"bits": s["out"][:, 0:6], "motion_depth": f[:, 6:10], "albedo": f[:, 10:13],
                "emission": f[:, 13:16]}
    g = s["graph"]
    g.run(s["sid"], s["cam"], s["size"], s["iterations"])
    return g.output("accumulate.out")


def _scene_size(kind, triangles):
    """(triangles traversed, bytes of the geometry and the environment, read once)"""
    if kind == "cornell":
        tess = max(1, round(math.sqrt(triangles / 1024)))
        return 1024 * tess * tess, 1024 * tess * tess * 84
    if kind == "soup":
        env = 2048 * 1024 if triangles >= 1_000_000 else 512 * 256
        return triangles, triangles * 84 + env * 16
    n = max(1, triangles // 50_000) * 50_000
    return n, n * 36 + 400 * 56 + 32 * 256 * 256 * 4 + 1024 * 512 * 16


# segments traced per sample, shadow rays included: measured means of the package's scenes
_SEGMENTS = {("cornell", True): 7.0, ("cornell", False): 4.0, ("soup", True): 3.3,
             ("soup", False): 2.6, ("instanced", True): 3.3, ("instanced", False): 2.6}


def _traced(kind, triangles, rays, shaded):
    """(bytes, flops) of tracing `rays` and shading `shaded` points: the eight boxes of one node
    per level of an 8-wide tree and two triangles per ray; a scene is read once at most."""
    n, size = _scene_size(kind, triangles)
    levels = max(1.0, math.log(n, 8))
    return (min(size, rays * (80 * levels + 2 * 84)),
            rays * (levels * 8 * 14 + 2 * 60) + shaded * 400)


def work(case):
    op = case["op"]
    if op in ("batch", "serve"):
        pool = _pool(case)
        b = f = 0.0
        samples = {}
        for i, w, h, spp in _mix(case):
            b += 16 * w * h
            samples[pool[i]] = samples.get(pool[i], 0) + w * h * spp
        for (kind, tris), n in samples.items():
            x = _traced(kind, tris, n * _SEGMENTS[(kind, True)], n * 2)
            b, f = b + x[0], f + x[1]
        return {"bytes": b, "flops": f}
    kind, tris = case["scene"], case["triangles"]
    if op == "rays":
        b, f = _traced(kind, tris, case["rays"], 0)
        return {"bytes": b + 64 * case["rays"], "flops": f}
    pix = case["width"] * case["height"]
    if op == "gbuffer":
        b, f = _traced(kind, tris, pix, pix)
        return {"bytes": b + 64 * pix, "flops": f}
    if op == "progressive":
        k = case["iterations"]
        b, f = _traced(kind, tris, pix * k * (1 + _SEGMENTS[(kind, True)]), pix * k * 3)
        return {"bytes": b + pix * k * (64 + 16 + 20 + 20 + 16), "flops": f}
    pix = case["pixels"] or pix
    seg = _SEGMENTS[(kind, case["nee"])]
    if case["length"] == 2:
        seg = min(seg, 3.0 if case["nee"] else 2.0)
    b, f = _traced(kind, tris, pix * case["spp"] * seg, pix * case["spp"] * (seg / 2 + 0.5))
    return {"bytes": b + 16 * pix, "flops": f}


def _room_triangles():
    """Positions of the 1,024-triangle room as the caller handed them over, in 64 bits."""
    data = S.cornell()
    v = torch.from_numpy(np.ascontiguousarray(data.vertices["position"])).cuda().double()
    first = np.zeros(data.triangle_count, np.int64)
    geoms = data.geometries
    for g in geoms:
        a, k = int(g["first_triangle"]), int(g["triangle_count"])
        first[a:a + k] = int(g["first_vertex"])
    idx = torch.from_numpy(data.indices.astype(np.int64) + first[:, None]).cuda()
    flags = np.zeros(data.triangle_count, np.int64)
    for g in geoms:
        a, k = int(g["first_triangle"]), int(g["triangle_count"])
        flags[a:a + k] = int(g["flags"])
    return v[idx], torch.from_numpy(flags).cuda()


def exact(case, seed):
    """Distances of closest-hit rays in the small room, by intersecting every triangle in 64 bits
    (double-sided or front-facing). The other outputs are Monte-Carlo images, whose samples are
    decided by comparisons that no other arithmetic repeats, ids and bits."""
    if case["op"] != "rays" or case["any"] or case["scene"] != "cornell" or \
            case["triangles"] != 1024:
        return None
    tri, flags = _room_triangles()
    rays = _rays(case, seed).double()
    p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    two = (flags & N.MESH_TWO_SIDED) != 0
    sign = torch.where((flags & N.MESH_FLIP_FACING) != 0, -1.0, 1.0).double()
    best = []
    for part in rays.split(8192):
        o, d = part[:, None, 0:3], part[:, None, 4:7]
        det = -(d * n).sum(-1)
        ao = o - p0
        t = (ao * n).sum(-1) / det
        dao = torch.linalg.cross(ao, d.expand_as(ao))
        u = (e2 * dao).sum(-1) / det
        v = -(e1 * dao).sum(-1) / det
        eps = 1e-9  # rays through a shared edge hit one of the two
        ok = (u >= -eps) & (v >= -eps) & (u + v <= 1 + eps) & (t >= 0) & (t <= part[:, 7:8])
        ok &= two | (det * sign > 0)
        t = torch.where(ok, t, torch.inf).amin(1)
        best.append(torch.where(torch.isinf(t), -1.0, t))
    return {"ids": None, "barycentrics": None, "t": torch.cat(best)}
