"""Long slices of the reference's random stream are generated by blocks that start a
jump of 512 refills apart, short ones and a context's first by one block.  Float
frames (a pixel's colour depends on the bits of its first sample) of a context
that has the jump equal those of contexts that walk from the seed: offsets and
lengths about one jump, between jumps and over many, skipped to, gone on from, and
restarted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REFILL = 624


@pytest.fixture(scope="module")
def setup(rtlib):
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=5, seed=2, res=24)
    frame = dict(frame, lights=[dict(frame["lights"][0], r=0.6)])

    def cam(w, h):
        return dict(frame, camera=scenes.look_at_camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, w, h))

    ctx = rtlib.Context(0)
    sc = rtlib.Scene(ctx, scene)
    end = sc.render_soft(cam(720, 720), 64)["stream_end"]
    assert end > 50000 * REFILL   # more refills than the jump costs
    yield sc, scene, cam
    ctx.close()


def check(rtlib, setup, w, h, samples, offset):
    sc, scene, cam = setup
    got = sc.render_soft(cam(w, h), samples, stream_offset=offset, want_float=True)
    fresh = rtlib.Context(0)
    want = rtlib.Scene(fresh, scene).render_soft(cam(w, h), samples, stream_offset=offset, want_float=True)
    fresh.close()
    assert got["stream_end"] == want["stream_end"]
    assert got["stream_end"] < 20000 * REFILL   # the fresh context has walked all of it
    assert np.array_equal(got["fimg"].view(np.uint32), want["fimg"].view(np.uint32))
    return got["stream_end"]


@pytest.mark.parametrize("refill", [0, 1, 511, 512, 513, 767, 768, 769, 1024, 4095, 20 * 512 + 77, 15000])
@pytest.mark.parametrize("size", [(40, 30, 2), (640, 400, 2), (701, 503, 2), (701, 503, 4)])
def test_slices(rtlib, setup, refill, size):
    check(rtlib, setup, *size, refill * REFILL + refill % 5 * 100)


@pytest.mark.parametrize("start", [0, 512 * REFILL - 1])
def test_consecutive(rtlib, setup, start):
    p = start
    for w, h, n in ((500, 400, 2), (30, 20, 2), (701, 503, 4), (333, 222, 3), (701, 503, 2)):
        p = check(rtlib, setup, w, h, n, p)
