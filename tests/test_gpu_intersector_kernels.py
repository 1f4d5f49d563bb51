"""Every kernel of either triangle test (RT_OPT_INTERSECTOR) is the one that
runs when that test is set.  The scenes are made of triangles so small that the
reference's test rejects them all (its determinant is below 1e-6: they have legs
of 5e-4) and the watertight one meets them: under the first test frames are all
background and rays meet nothing, under the second

  A   a patch below the camera is seen,
  B   a patch between A and a lamp keeps the lamp from what the camera sees,
  C   a patch behind the camera is seen in A's reflections, and A keeps a lamp
      below it from what is seen there,

so that camera rays, shadow rays, mirrored rays and their shadow rays each show
which test their kernel has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LEG = 5.0e-4
PATCHES = {"A": (-0.006, -0.006, 24, 24, 0.0), "B": (0.002, -0.002, 8, 8, 0.004), "C": (-0.008, -0.008, 32, 32, 0.05)}


def scene_of(names):
    verts, tris = [], []
    for k in names:
        x0, y0, nx, ny, z = PATCHES[k]
        at = sum(len(v) for v in verts)
        gy, gx = np.mgrid[0:ny + 1, 0:nx + 1]
        verts.append(np.stack([x0 + LEG * gx, y0 + LEG * gy, np.full_like(gx, z, dtype=np.float64)], -1).reshape(-1, 3))
        c = (np.arange(ny)[:, None] * (nx + 1) + np.arange(nx)).ravel() + at
        tris.append(np.stack([np.stack([c, c + 1, c + nx + 2], -1), np.stack([c, c + nx + 2, c + nx + 1], -1)], 1).reshape(-1, 3))
    v = np.concatenate(verts).astype(np.float32)
    return {"verts": v, "tris": np.concatenate(tris).astype(np.int32),
            "vattr": np.full(v.shape, 0.8, np.float32), "flags": np.zeros(sum(len(t) for t in tris), np.uint32)}


def frame_of(rf=0.0, ns=5.0):
    from raptor_gb300 import scenes
    cam = scenes.look_at_camera((0.0, 0.0, 0.02), (0.0, 0.0, 0.0), 5.72, 21, 19, background=(110.0, 160.0, 230.0))
    return {"camera": cam, "lights": [], "material": {"ka": (30.0, 40.0, 50.0), "kd": (100.0, 100.0, 100.0),
                                                      "ks": (20.0, 20.0, 20.0), "ns": ns, "rf": rf}}


def lamp(pos):
    from raptor_gb300 import scenes
    return dict(scenes.point_light(pos), r=0.0)


def rendered(rtlib, ctx, kind, names, lights):
    scene = scene_of(names)
    f = dict(frame_of(rf=0.4 if kind in ("tree", "reference", "pixel") else 0.0,
                      ns=20.5 if kind == "aa power" else 5.0), lights=lights)
    H, W = f["camera"]["yres"], f["camera"]["xres"]
    ao = {"samples": 5, "dist": 0.1, "seed": 3}
    if kind.startswith("batch"):
        b = rtlib.Batch(ctx)
        i = b.add_scene(scene)
        b.build()
        rgb = torch.zeros((H, W, 3), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        b.set_jobs([rtlib.make_job(i, dict(f, ao=ao) if "ao" in kind else f, rgb)])
        if "wave" in kind:
            b.set_config(kernel=rtlib.RT_KERNEL_WAVE)
        b.render()
        out = rgb.cpu().numpy()
        b.close()
        return out
    sc = rtlib.Scene(ctx, scene)
    if "wave" in kind:
        ctx.set_option(rtlib.RT_OPT_RENDER_KERNEL, rtlib.RT_KERNEL_WAVE)
    if "ao" in kind:
        out = sc.render(dict(f, ao=ao))["rgb"]
    elif kind == "table":
        out = sc.render(dict(f, materials=[f["material"]]))["rgb"]
    elif kind == "image":
        out = sc.render_image(f)["fimg"]
    elif kind == "tone":
        out = sc.render_tone_mapped(f, {"mode": 5})["rgb"]
    elif kind == "aa loop":
        out = sc.render_aa(f, 6, 6)["rgb"]
    elif kind.startswith("aa"):
        out = sc.render_aa(f, 2, 2)["rgb"]
    elif kind == "soft":
        out = sc.render_soft(dict(f, lights=[dict(l, r=0.001) for l in lights]), 4)["rgb"]
    elif kind == "reference":
        out = sc.render_distributed(dict(f, lights=[dict(l, r=0.001) for l in lights]), soft=4)["rgb"]
    elif kind == "pixel":
        out = sc.render_distributed(f, soft=1, stream=rtlib.RT_STREAM_PIXEL, seed=2)["rgb"]
    elif kind == "float":
        img = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
        sc.render_float(f, img)
        out = img.cpu().numpy()
    else:
        out = sc.render(f)["rgb"]
    ctx.set_option(rtlib.RT_OPT_RENDER_KERNEL, rtlib.RT_KERNEL_PIXEL)
    sc.close()
    return out


def both(rtlib, kind, names, lights):
    """The frame under the watertight test; under the other it is one colour."""
    ctx = rtlib.Context(0)
    one = rendered(rtlib, ctx, kind, names, lights)
    assert (one == one[0, 0]).all()
    ctx.set_option(rtlib.RT_OPT_INTERSECTOR, rtlib.RT_ISECT_WATERTIGHT)
    wt = rendered(rtlib, ctx, kind, names, lights)
    ctx.close()
    return wt, one


KINDS = ["plain", "table", "image", "tone", "aa", "aa loop", "aa power", "tree", "soft", "reference", "pixel", "float",
         "wave", "batch", "batch wave"]


@pytest.mark.parametrize("kind", KINDS)
def test_camera_and_shadow_rays(rtlib, kind):
    L = [lamp((1.0, 0.0, 1.0))]
    lit, background = both(rtlib, kind, "A", L)
    dark = both(rtlib, kind, "A", [])[0]
    shadowed = both(rtlib, kind, "AB", L)[0]
    if kind != "tone":   # its colours depend on the whole frame's
        assert (lit != background).any(-1).all() and (dark != background).any(-1).all()
        assert (lit != dark).any(-1).all()
        assert np.array_equal(shadowed, dark)
    else:
        assert not np.array_equal(lit, background) or not np.array_equal(dark, background)


@pytest.mark.parametrize("kind", ["tree", "reference", "pixel"])
def test_mirrored_rays(rtlib, kind):
    dark = both(rtlib, kind, "A", [])[0]
    behind = both(rtlib, kind, "AC", [])[0]
    assert (behind != dark).any(-1).all()
    lit = both(rtlib, kind, "AC", [lamp((1.0, 0.0, -0.5))])[0]
    assert (lit != behind).any(-1).all()
    below = both(rtlib, kind, "AC", [lamp((0.0, 0.0, -1.0))])[0]
    assert np.array_equal(below, behind)


@pytest.mark.parametrize("kind", ["ao", "wave ao", "batch ao", "batch wave ao"])
def test_ambient_rays(rtlib, kind):
    """C is a lid of 3 % of A's sky: rays that meet nothing leave both frames alike."""
    open_, background = both(rtlib, kind, "A", [])
    lid = both(rtlib, kind, "AC", [])[0]
    assert (open_ != background).any(-1).all()
    assert not np.array_equal(lid, open_)


@pytest.mark.parametrize("n", [1000, 200000, -1])
def test_rays(rtlib, n):
    """Few rays, the work queue, and (-1) the list of scattered any-hit rays; from
    host memory too where it takes another way."""
    n = 4 * 8 * 128 * torch.cuda.get_device_properties(0).multi_processor_count if n < 0 else n
    rng = np.random.default_rng(3)
    o = np.concatenate([rng.uniform(-0.005, 0.005, (n, 2)), rng.uniform(0.01, 0.04, (n, 1))], 1)
    to = np.concatenate([rng.uniform(-0.005, 0.005, (n, 2)), np.zeros((n, 1))], 1)
    d = to - o
    dist = np.linalg.norm(d, axis=1)
    rays = rtlib.rays_array(o.astype(np.float32), (d / dist[:, None]).astype(np.float32), (2.0 * dist).astype(np.float32))
    dev = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for option, met in ((rtlib.RT_ISECT_REFERENCE, 0), (rtlib.RT_ISECT_WATERTIGHT, 1)):
        ctx = rtlib.Context(0)
        ctx.set_option(rtlib.RT_OPT_INTERSECTOR, option)
        sc = rtlib.Scene(ctx, scene_of("A"))
        sc.closest_into(dev, hits)
        rtlib._check(rtlib.lib().rt_trace_any(sc.h, rtlib.ptr(dev), n, rtlib.ptr(occ)))
        assert ((hits[:, 0] >= 0) == bool(met)).all() and (occ == met).all()
        assert ((sc.closest(rays)["tri"] >= 0) == bool(met)).all() and (sc.any(rays) == met).all()
        if n <= 16384:
            no_alloc = np.zeros(n, rtlib.HIT_DTYPE)
            rtlib._check(rtlib.lib().rt_trace_closest_noalloc(sc.h, rtlib.ptr(rays), n, rtlib.ptr(no_alloc)))
            assert ((no_alloc["tri"] >= 0) == bool(met)).all()
        ctx.close()


def test_gradients(rtlib):
    f = dict(frame_of(), lights=[lamp((1.0, 0.0, 1.0))])
    for names, option, some in (("A", rtlib.RT_ISECT_REFERENCE, False), ("A", rtlib.RT_ISECT_WATERTIGHT, True),
                                ("AB", rtlib.RT_ISECT_WATERTIGHT, False)):
        ctx = rtlib.Context(0)
        ctx.set_option(rtlib.RT_OPT_INTERSECTOR, option)
        scene = scene_of(names)
        sc = rtlib.Scene(ctx, scene)
        one = torch.ones((f["camera"]["yres"], f["camera"]["xres"], 3), device="cuda")
        gpos, gcol = (torch.full(scene["verts"].shape, 9.0, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        sc.render_adjoint(f, one, gpos, gcol)
        assert bool((gcol != 0).any()) == some
        ctx.close()
