"""Device memory that distributed frames on per-pixel streams keep: the rays of
the camera rays' sets and the nodes below them that such a frame can have, not
what the largest could."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# Rays of the sets (items): at most 2 sets a pixel of `diffuse` rays, here a set
# for three quarters of the pixels at most.  Bytes an item: its record and colour
# and sets in lists of twice the longer set's (2 * 9/8 * (48 + 32)) and its hit (52);
# a node: 132.  With a quarter as headroom, and 64 MB for the rest.
@pytest.mark.parametrize("glass,diffuse,nodes", [(False, 16, 0), (True, 0, 2), (True, 4, 2), (True, 8, 3)])
def test_held(rtlib, glass, diffuse, nodes):
    from raptor_gb300 import scenes
    scene, frame = scenes.glass_scene(freq=16, res=64)
    size = 400
    cam = scenes.look_at_camera((0.3, 0.8, 4.0), (0.0, -0.2, 0.0), 50.0, size, size, background=(110.0, 160.0, 230.0))
    mats = [dict(frame["materials"][0], rfd=0.1), dict(frame["materials"][1], rfd=0.1, td=0.05)]
    if not glass:
        mats[1] = dict(mats[1], tran=0.0, rf=0.2)
    # the driver's stacks for these kernels, kept for the process, come with a first frame
    first = rtlib.Context(0)
    rtlib.Scene(first, scene).render_distributed(dict(frame, materials=mats), soft=1, diffuse=diffuse,
                                                 stream=rtlib.RT_STREAM_PIXEL, seed=5)
    first.close()
    frame = dict(frame, camera=cam, materials=mats)
    ctx = rtlib.Context(0)
    sc = rtlib.Scene(ctx, scene)
    rgb = torch.empty((size, size, 3), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    out = sc.render_distributed(frame, soft=1, diffuse=diffuse, stream=rtlib.RT_STREAM_PIXEL, seed=5, rgb=rgb)
    held = before - torch.cuda.mem_get_info()[0]
    items = size * size * max(diffuse, 1) * (2.0 if glass else 0.9)
    assert out["stats"].status == 0
    assert held < 1.25 * items * (2 * 9 / 8 * 80 + 52 + 132 * nodes) + 64e6, (held, items)
    ctx.close()
