"""Every frame kind is compiled once per triangle test (RT_OPT_INTERSECTOR):
each dispatch must reach the kernels of the test that is set.  The two tests
accept the same hits but within rounding of an edge, and their distances
differ in the last bits, so a frame of either agrees with the other's on all
but a few pixels (at least 99 % of them, within 2 levels), while the float
frames, whose barycentrics come from different arithmetic, are not all
equal bit for bit -- which shows that the option reached the kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def frames(rtlib, sc, ctx, kind, frame):
    H, W = frame["camera"]["yres"], frame["camera"]["xres"]
    if kind == "ao":
        return sc.render(dict(frame, ao={"samples": 5, "dist": 2.0, "seed": 3}))["rgb"]
    if kind == "aa":
        return sc.render_aa(frame, 2, 2)["rgb"]
    if kind == "tree":
        return sc.render(dict(frame, material=dict(frame["material"], rf=0.4)))["rgb"]
    if kind == "tone":
        return sc.render_tone_mapped(frame, {"mode": 5})["rgb"]
    if kind == "soft":
        lights = [dict(frame["lights"][0], r=0.5)]
        return sc.render_soft(dict(frame, lights=lights), 4)["rgb"]
    if kind == "diffuse":
        mat = dict(frame["material"], rf=0.3, rfd=0.1)
        return sc.render_distributed(dict(frame, material=mat), soft=4, diffuse=4, stream=rtlib.RT_STREAM_PIXEL,
                                     seed=2)["rgb"]
    if kind == "float":
        img = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
        sc.render_float(frame, img)
        return img.cpu().numpy()
    if kind == "wave":
        ctx.set_option(rtlib.RT_OPT_RENDER_KERNEL, rtlib.RT_KERNEL_WAVE)
        out = sc.render(frame)["rgb"]
        ctx.set_option(rtlib.RT_OPT_RENDER_KERNEL, rtlib.RT_KERNEL_PIXEL)
        return out
    return sc.render(frame)["rgb"]


@pytest.mark.parametrize("kind", ["plain", "ao", "aa", "tree", "tone", "soft", "diffuse", "float", "wave"])
def test_dispatch(rtlib, kind):
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=9, seed=4, res=61)
    c = rtlib.Context(0)
    sc = rtlib.Scene(c, scene)
    ref = frames(rtlib, sc, c, kind, frame)
    c.set_option(rtlib.RT_OPT_INTERSECTOR, rtlib.RT_ISECT_WATERTIGHT)
    wt = frames(rtlib, sc, c, kind, frame)
    far = np.abs(ref.astype(np.float64) - wt.astype(np.float64)).max(-1) > 2
    assert far.mean() < 0.01
    if kind == "float":
        assert not np.array_equal(ref, wt)
    sc.close()
    c.close()
