"""Workloads by which the ray-tracing core is timed.

Each case is one thing a program does with the library, called through
raptor_gb300.core: rays traced against a built scene, frames of every kind the
library renders, a moving scene's rebuild or refit with its frame, a step of
an inverse-rendering loop, and a batch of small scenes.  Scenes are the seeded
synthetic ones of raptor_gb300.scenes (sphere on a ground, diamond-square
terrain, instanced spheres and cubes, glass sphere); sizes are the benchmark's
and the tests', and odd ones between them.

`prepare` leaves the scene uploaded and its hierarchy built, with output
buffers on the device, as a renderer keeps them between frames; a case's `run`
is the call or calls a program makes for one frame or one query.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from raptor_gb300 import core, scenes


# ------------------------------------------------------------------ cases

def listed():
    return [
        # a picking or physics query: a few hundred rays in host memory against
        # a small mesh, hits back in host memory; latency is all of it
        {"name": "query-rays-300", "kind": "closest", "scene": "sphere", "size": 32, "rays": 300, "host": True},
        # a visibility pass of another program: incoherent any-hit rays already
        # on the device
        {"name": "visibility-rays-2M", "kind": "any", "scene": "terrain", "size": 700, "rays": 2000003, "host": False},
        # an interactive preview: small mesh, small frame, one light
        {"name": "sphere-512", "kind": "frame", "scene": "sphere", "size": 32, "xres": 512, "yres": 512},
        # the large single frame: two million triangles, full HD, sun shadows
        {"name": "terrain-1080p", "kind": "frame", "scene": "terrain", "size": 1024, "xres": 1920, "yres": 1080},
        # a final frame: anti-aliased and tone mapped, odd resolution
        {"name": "terrain-aa-tone", "kind": "tone", "scene": "terrain", "size": 725, "xres": 1283, "yres": 717,
         "aa_x": 2, "aa_y": 2, "mode": 5, "gamma": 2.2},
        # ambient occlusion over many separate objects: short incoherent rays
        {"name": "instances-ao-720p", "kind": "ao", "scene": "instances", "size": 2000, "xres": 1280, "yres": 720,
         "samples": 16},
        # mirrors and refraction: a tree of rays per pixel
        {"name": "glass-tree-512", "kind": "tree", "scene": "glass", "size": 32, "xres": 512, "yres": 512},
        # an animation with soft shadows: every frame draws on from where the
        # last one ended in the reference's random stream
        {"name": "terrain-soft-900p", "kind": "soft", "scene": "terrain", "size": 725, "xres": 1600, "yres": 900,
         "samples": 16},
        # diffuse reflections and refractions, the heaviest kind of frame
        {"name": "glass-diffuse-512", "kind": "diffuse", "scene": "glass", "size": 32, "xres": 512, "yres": 512,
         "soft": 16, "diffuse": 16},
        # a simulation that moves every vertex: rebuild, then a frame
        {"name": "terrain-rebuild-480p", "kind": "rebuild", "scene": "terrain", "size": 1024, "xres": 854, "yres": 480},
        # a step of an inverse-rendering loop: new vertices and colours, float
        # frame, gradients of an L2 loss
        {"name": "adjoint-step-256", "kind": "adjoint", "scene": "bumpy", "size": 50, "xres": 256, "yres": 256},
        # many small scenes of mixed sizes, resolutions and ray mixes in one launch
        {"name": "batch-24", "kind": "batch", "scene": "mixed", "size": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "any", "frame", "frame", "aa", "tone", "ao", "tree", "soft", "diffuse", "rebuild",
                       "refit", "adjoint", "batch"])
    if kind == "batch":
        return {"kind": kind, "scene": "mixed", "size": _log(rng, 2, 24)}
    if kind == "adjoint":
        return {"kind": kind, "scene": "bumpy", "size": _log(rng, 6, 50), "xres": _log(rng, 48, 256),
                "yres": _log(rng, 48, 256)}
    scene = {"ao": "instances", "tree": "glass", "diffuse": "glass", "rebuild": "terrain", "refit": "terrain"}.get(kind)
    scene = scene or rng.choice(["sphere", "terrain", "terrain"])
    top = {"sphere": 64, "terrain": 1024, "instances": 2000, "glass": 40}[scene]
    case = {"kind": kind, "scene": scene, "size": _log(rng, max(4, top // 32), top)}
    if kind in ("closest", "any"):
        case.update(rays=_log(rng, 1, 2000000), host=rng.random() < 0.4)
        return case
    w, h = {"tree": (640, 512), "diffuse": (400, 400), "tone": (1283, 717), "aa": (1283, 717),
            "soft": (1600, 900)}.get(kind, (1920, 1080))
    s = math.exp(rng.uniform(math.log(0.05), 0.0))
    case.update(xres=max(17, int(w * s)), yres=max(13, int(h * s * rng.uniform(0.7, 1.0))))
    if kind == "frame":
        case.update(spot=rng.random() < 0.3)
    if kind in ("aa", "tone"):
        case.update(aa_x=rng.randint(1, 3), aa_y=rng.randint(1, 2))
    if kind == "tone":
        case.update(mode=rng.choice([4, 5, 6, 7]), gamma=rng.choice([1.0, 2.2]))
    if kind in ("ao", "soft"):
        case.update(samples=rng.choice([1, 4, 7, 16]))
    if kind == "diffuse":
        case.update(soft=rng.choice([1, 4, 16]), diffuse=rng.choice([0, 4, 16]))
    return case


# ----------------------------------------------------------------- scenes

def _mesh(case, seed):
    """Scene and frame dicts (raptor_gb300.scenes) of a case."""
    kind, n = case["scene"], int(case["size"])
    if kind == "sphere":
        scene, frame = scenes.icosphere_scene(freq=n, seed=seed, res=64)
        eye, at, fov, bg = (0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, (0.0, 0.0, 0.0)
    elif kind == "terrain":
        size = 1 << max(2, (n - 1).bit_length())
        extent = 1024.0 * n / size
        scene, frame = scenes.terrain_scene(size_pow2=size, seed=seed, crop=n + 1 if n < size else 0)
        eye, at, fov, bg = (0.0, 300.0, 0.0), (extent / 2, 100.0, extent / 2), 60.0, (110.0, 160.0, 230.0)
    elif kind == "instances":
        scene, frame = scenes.instances_scene(n_inst=n, seed=seed)
        eye, at, fov, bg = (50.0, 50.0, -40.0), (50.0, 50.0, 50.0), 60.0, (0.0, 0.0, 0.0)
    elif kind == "glass":
        scene, frame = scenes.glass_scene(freq=n, res=64, seed=seed)
        eye, at, fov, bg = (0.3, 0.8, 4.0), (0.0, -0.2, 0.0), 50.0, (110.0, 160.0, 230.0)
    else:   # bumpy: the displaced sphere of the inverse-rendering loop
        scene, _, frame = scenes.adjoint_scene(freq=n, seed=seed, res=64)
        eye, at, fov, bg = (0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 40.0, (0.0, 0.0, 0.0)
    if "xres" in case:
        frame = dict(frame, camera=scenes.look_at_camera(eye, at, fov, case["xres"], case["yres"], background=bg))
    return scene, frame


def _rays(scene, n, seed, aimed):
    """Rays from random points above the scene towards random points of its
    surface (aimed) or of its box, in no order: the first all hit, the second
    hit or miss."""
    rng = np.random.default_rng(seed + 77)
    lo, hi = scene["verts"].min(0).astype(np.float64), scene["verts"].max(0).astype(np.float64)
    ext = np.maximum(hi - lo, 1e-3)
    o = lo + ext * rng.uniform(-0.2, 1.2, (n, 3))
    o[:, 1] = hi[1] + ext[1] * rng.uniform(0.05, 0.5, n)
    if aimed:
        tri = scene["tris"][rng.integers(0, scene["tris"].shape[0], n)]
        w = rng.dirichlet((2.0, 2.0, 2.0), n)
        to = (scene["verts"][tri].astype(np.float64) * w[:, :, None]).sum(1)
    else:
        to = lo + ext * rng.uniform(0.0, 1.0, (n, 3))
    d = to - o
    dist = np.sqrt((d * d).sum(1))
    return core.rays_array(o.astype(np.float32), (d / dist[:, None]).astype(np.float32), dist.astype(np.float32))


def prepare(case, seed):
    kind = case["kind"]
    ctx = core.Context(0)
    st = {"case": case, "ctx": ctx}
    if kind == "batch":
        items = scenes.batched_scenes(n=case["size"], seed=3, tri_hi=200000)
        rng = np.random.default_rng(seed)
        for s, _ in items:   # the same mix of sizes, other shapes and colours
            s["verts"] = (s["verts"] * rng.uniform(0.9, 1.1, 3)).astype(np.float32)
            s["vattr"] = rng.random(s["vattr"].shape, dtype=np.float32)
        b = core.Batch(ctx)
        idx = [b.add_scene(s) for s, _ in items]
        b.build()
        st["rgb"] = [torch.empty((f["camera"]["yres"], f["camera"]["xres"], 3), dtype=torch.uint8, device="cuda")
                     for _, f in items]
        b.set_jobs([core.make_job(i, f, buf) for i, (_, f), buf in zip(idx, items, st["rgb"])])
        st["batch"] = b
        return st
    scene, frame = _mesh(case, seed)
    if kind in ("closest", "any"):
        rays = _rays(scene, case["rays"], seed, kind == "closest")
        st["scene"] = core.Scene(ctx, scene)
        if case["host"]:
            st["rays"] = rays
        else:
            st["rays"] = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
            words = (case["rays"], 4) if kind == "closest" else (case["rays"],)
            st["out"] = torch.empty(words, dtype=torch.int32 if kind == "closest" else torch.uint8, device="cuda")
            torch.cuda.synchronize()
        return st
    H, W = frame["camera"]["yres"], frame["camera"]["xres"]
    st["scene"] = sc = core.Scene(ctx, scene)
    st["rgb"] = torch.empty((H, W, 3), dtype=torch.uint8, device="cuda")
    st["ids"] = torch.empty((H, W), dtype=torch.int32, device="cuda")
    rng = np.random.default_rng(seed + 5)
    if kind == "frame" and case.get("spot"):
        p = np.asarray(frame["camera"]["pos"]) + np.asarray([1.0, 2.0, 0.5])
        frame = dict(frame, lights=frame["lights"] + [scenes.spot_light(p, frame["camera"]["z_axis"], 0.1, 0.5)])
    elif kind == "tone":
        st["tone"] = {"mode": case["mode"], "gamma": case["gamma"]}
    elif kind == "ao":
        frame = dict(frame, ao={"samples": case["samples"], "dist": 5.0, "seed": seed & 0xffff})
    elif kind == "soft":
        span = float(np.ptp(scene["verts"][:, 0]))
        top = float(scene["verts"][:, 1].max())
        lamp = dict(scenes.point_light((0.4 * span, top + 0.3 * span, 0.3 * span)), r=0.04 * span)
        frame = dict(frame, lights=[lamp, scenes.directional_light((-0.4, -0.8, -0.3), rgb=(120.0, 120.0, 110.0))])
        st["offset"] = 0
    elif kind == "diffuse":
        lights = [dict(frame["lights"][0], r=0.7), frame["lights"][1]]
        mats = [dict(frame["materials"][0], rfd=0.2), dict(frame["materials"][1], rfd=0.1, td=0.05)]
        frame = dict(frame, lights=lights, materials=mats, material=mats[0])
        st["seed"] = seed
    elif kind in ("rebuild", "refit"):
        v = scene["verts"] + rng.normal(0.0, 0.05, scene["verts"].shape).astype(np.float32)
        st["verts"] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
        torch.cuda.synchronize()
    elif kind == "adjoint":
        # the library on torch's stream: the loss between its two calls is torch's
        st["stream"] = torch.cuda.Stream()
        ctx.set_stream(st["stream"].cuda_stream)
        st["verts"], st["cols"] = torch.from_numpy(scene["verts"]).cuda(), torch.from_numpy(scene["vattr"]).cuda()
        st["target"] = torch.from_numpy(rng.uniform(0.0, 255.0, (H, W, 3)).astype(np.float32)).cuda()
        st["img"] = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
        st["gpos"], st["gcol"] = torch.empty_like(st["verts"]), torch.empty_like(st["cols"])
        torch.cuda.synchronize()
    st["frame"] = frame
    return st


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "batch":
        st["batch"].render()
        return st["rgb"]
    sc = st["scene"]
    if kind == "closest":
        if case["host"]:
            h = sc.closest(st["rays"])
            return {"id": h["tri"], "t": h["t"], "u": h["u"], "v": h["v"]}
        sc.closest_into(st["rays"], st["out"])
        f = st["out"].view(torch.float32)
        return {"id": st["out"][:, 0], "t": f[:, 1], "u": f[:, 2], "v": f[:, 3]}
    if kind == "any":
        if case["host"]:
            return sc.any(st["rays"])
        core._check(core.lib().rt_trace_any(sc.h, core.ptr(st["rays"]), case["rays"], core.ptr(st["out"])))
        return st["out"]
    frame, rgb, ids = st["frame"], st["rgb"], st["ids"]
    if kind in ("frame", "ao", "tree"):
        sc.render(frame, rgb=rgb, ids=ids)
    elif kind == "aa":
        sc.render_aa(frame, case["aa_x"], case["aa_y"], rgb=rgb)
        return rgb
    elif kind == "tone":
        sc.render_tone_mapped(frame, st["tone"], aa=(case["aa_x"], case["aa_y"]), rgb=rgb)
        return rgb
    elif kind == "soft":
        r = sc.render_soft(frame, case["samples"], stream_offset=st["offset"], rgb=rgb)
        st["offset"] = r["stream_end"]
        return {"rgb": rgb, "stream_end": r["stream_end"]}
    elif kind == "diffuse":
        r = sc.render_distributed(frame, soft=case["soft"], diffuse=case["diffuse"], stream=core.RT_STREAM_PIXEL,
                                  seed=st["seed"], rgb=rgb)
        return {"rgb": rgb, "numbers": r["stream_end"]}
    elif kind in ("rebuild", "refit"):
        if kind == "rebuild":
            sc.update_vertices(st["verts"])
        else:
            sc.refit_vertices(st["verts"])
        sc.render(frame, rgb=rgb, ids=ids)
    elif kind == "adjoint":
        with torch.cuda.stream(st["stream"]):
            sc.update_vertices(st["verts"])
            sc.update_attributes(st["cols"])
            sc.render_float(frame, st["img"], ids)
            sc.render_adjoint(frame, 2.0 * (st["img"] - st["target"]), st["gpos"], st["gcol"])
        return {"img": st["img"], "ids": ids, "gpos": st["gpos"], "gcol": st["gcol"]}
    return {"rgb": rgb, "ids": ids}


# ------------------------------------------------------------------- work

def _triangles(case):
    n = case["size"]
    return {"sphere": 20 * n * n + 2, "terrain": 2 * n * n, "instances": 2000 * n, "glass": 40 * n * n + 2,
            "bumpy": 20 * n * n, "mixed": 40000 * n}[case["scene"]]


def work(case):
    """Bytes: the mesh as uploaded (vertices, colours and indices, about 24
    bytes a triangle) and the rays read once, the outputs written once.
    Operations: per ray, one 6-plane box test of 8 children on each level of
    an 8-wide tree, three triangle tests and, for a hit, its shading."""
    kind, nt = case["kind"], _triangles(case)
    levels = max(1.0, math.log(max(nt, 8) / 3.0, 8.0))
    per_ray = levels * 8 * 18 + 3 * 50 + 60
    if kind in ("closest", "any"):
        n = case["rays"]
        return {"bytes": 24 * nt + n * (32 + (16 if kind == "closest" else 1)), "flops": n * per_ray}
    if kind == "batch":
        pix = case["size"] * 6e5
        return {"bytes": 24 * nt + 3 * pix, "flops": 3 * pix * per_ray}
    pix = case["xres"] * case["yres"]
    rays = {"ao": 1 + 0.8 * case.get("samples", 0), "soft": 1.5 + 0.5 * case.get("samples", 0), "tree": 6.0,
            "diffuse": 10 + 0.7 * case.get("soft", 1) * max(case.get("diffuse", 0), 1), "adjoint": 2.5,
            "aa": 1.5, "tone": 1.5}.get(kind, 1.5) * case.get("aa_x", 1) * case.get("aa_y", 1)
    out = {"adjoint": 16 * pix + 24 * nt, "soft": 3 * pix, "diffuse": 3 * pix, "aa": 3 * pix, "tone": 3 * pix}
    moved = 6 * nt if kind in ("rebuild", "refit") else 0
    return {"bytes": 24 * nt + moved + out.get(kind, 7 * pix), "flops": rays * pix * per_ray}


# ------------------------------------------------------- 64-bit references

def _first_hits(V, T, o, d, tmax, eps=1e-3):
    """Closest hit of every ray by testing every triangle in 64 bits (torch):
    id (-1: none), t, u (weight of c), v (weight of b)."""
    A, B, Cv = V[T[:, 0]], V[T[:, 1]], V[T[:, 2]]
    e1, e2 = Cv - A, B - A
    n, step = o.shape[0], max(1, 30000000 // max(1, T.shape[0]))
    ids = torch.full((n,), -1, dtype=torch.int64, device=V.device)
    out = torch.zeros((n, 3), dtype=torch.float64, device=V.device)
    for k in range(0, n, step):
        D, O = d[k:k + step, None, :], o[k:k + step, None, :]
        P = torch.linalg.cross(D.expand(-1, T.shape[0], -1), e2[None].expand(D.shape[0], -1, -1))
        det = (e1[None] * P).sum(-1)
        S = O - A[None]
        u = (S * P).sum(-1) / det
        Q = torch.linalg.cross(S, e1[None].expand(D.shape[0], -1, -1))
        v = (D * Q).sum(-1) / det
        t = (e2[None] * Q).sum(-1) / det
        ok = (det.abs() >= 1e-6) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > eps) & (t < tmax[k:k + step, None])
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, at = t.min(1)
        hit = torch.isfinite(best)
        ids[k:k + step] = torch.where(hit, at, torch.full_like(at, -1))
        g = at[:, None]
        out[k:k + step] = torch.cat([best[:, None], u.gather(1, g), v.gather(1, g)], 1) * hit[:, None]
    out[ids < 0] = 0.0
    return ids, out[:, 0], out[:, 1], out[:, 2]


def _camera_rays(cam, device):
    """Rays of every pixel, row by row, from the camera's 32-bit numbers."""
    f = lambda k: torch.tensor([float(np.float32(x)) for x in cam[k]], dtype=torch.float64, device=device)  # noqa: E731
    W, H = cam["xres"], cam["yres"]
    w, h = np.float32(cam["w"]), np.float32(cam["h"])
    xt = torch.arange(W, dtype=torch.float64, device=device) * float(w * np.float32(2.0) / np.float32(W)) - float(w)
    yt = torch.arange(H, dtype=torch.float64, device=device) * float(h * np.float32(2.0) / np.float32(H)) - float(h)
    d = xt[None, :, None] * f("x_axis") + yt[:, None, None] * f("y_axis") + cam["t"] * f("z_axis")
    d = d / d.norm(dim=-1, keepdim=True)
    return f("pos").expand(H * W, 3), d.reshape(-1, 3)


def exact(case, seed):
    """Hits of the ray queries and the float frame and gradients of the
    inverse-rendering step, by brute force and autograd in 64 bits, where that
    is quick; frames in bytes have no such value."""
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "closest":
        if case["rays"] * _triangles(case) > 4e9:
            return None
        scene, _ = _mesh(case, seed)
        rays = _rays(scene, case["rays"], seed, kind == "closest")
        V, T = torch.from_numpy(scene["verts"]).double().to(dev), torch.from_numpy(scene["tris"]).long().to(dev)
        o, d = torch.from_numpy(rays["o"].astype(np.float64)).to(dev), torch.from_numpy(rays["d"].astype(np.float64)).to(dev)
        ids, t, u, v = _first_hits(V, T, o, d, torch.full((o.shape[0],), math.inf, dtype=torch.float64, device=dev))
        t = torch.where(ids >= 0, t, torch.full_like(t, float(np.finfo(np.float32).max)))
        return {"id": None, "t": t, "u": u, "v": v}
    if kind != "adjoint" or case["xres"] * case["yres"] * _triangles(case) > 4e9:
        return None
    scene, frame = _mesh(case, seed)
    H, W = case["yres"], case["xres"]
    target = np.random.default_rng(seed + 5).uniform(0.0, 255.0, (H, W, 3)).astype(np.float32)
    V = torch.from_numpy(scene["verts"]).double().to(dev).requires_grad_(True)
    C = torch.from_numpy(scene["vattr"]).double().to(dev).requires_grad_(True)
    T = torch.from_numpy(scene["tris"]).long().to(dev)
    o, d = _camera_rays(frame["camera"], dev)
    mat, light = frame["material"], frame["lights"][0]
    vec = lambda x: torch.tensor([float(np.float32(q)) for q in x], dtype=torch.float64, device=dev)  # noqa: E731
    with torch.no_grad():
        ids, _, _, _ = _first_hits(V, T, o, d, torch.full((o.shape[0],), math.inf, dtype=torch.float64, device=dev))
    hit = torch.nonzero(ids >= 0)[:, 0]
    tri, o, d = T[ids[hit]], o[hit], d[hit]
    A, B, Cv = V[tri[:, 0]], V[tri[:, 1]], V[tri[:, 2]]
    e1, e2 = Cv - A, B - A
    P = torch.linalg.cross(d, e2)
    det = (e1 * P).sum(-1)
    Q = torch.linalg.cross(o - A, e1)
    u, v, t = ((o - A) * P).sum(-1) / det, (d * Q).sum(-1) / det, (e2 * Q).sum(-1) / det
    p = o + t[:, None] * d
    n = torch.linalg.cross(e2, e1)
    n = n / n.norm(dim=-1, keepdim=True)
    n = torch.where(((n * d).sum(-1) > 0)[:, None], -n, n)
    to = vec(light["pos"]) - p
    dist = to.norm(dim=-1)
    ldir = to / dist[:, None]
    with torch.no_grad():
        blocked = _first_hits(V, T, p, ldir, dist)[0] >= 0
    s = (ldir * n).sum(-1)
    r = (d * (ldir - 2.0 * s[:, None] * n)).sum(-1)
    spec = torch.where(r > 0, r.clamp(min=1e-300) ** mat["ns"], torch.zeros_like(r))
    col = (u[:, None] * C[tri[:, 2]] + v[:, None] * C[tri[:, 1]] + (1.0 - u - v)[:, None] * C[tri[:, 0]]) * vec(mat["kd"])
    lit = (~blocked & (s >= 0)).double()[:, None]
    c = vec(mat["ka"]) + lit * vec(light["rgb"]) / 255.0 * (s[:, None] * col + spec[:, None] * vec(mat["ks"]))
    img = vec(frame["camera"]["background"]).expand(H * W, 3).clone()
    img[hit] = c
    tgt = torch.from_numpy(target).double().to(dev).reshape(-1, 3)
    ((img - tgt) ** 2).sum().backward()
    return {"img": img.detach().reshape(H, W, 3), "ids": None, "gpos": V.grad, "gcol": C.grad}
