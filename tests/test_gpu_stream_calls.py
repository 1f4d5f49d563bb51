"""What a frame on the reference's random stream leaves behind: nothing that still
runs on the device, and a generator from whose position, or the words before it,
the next frame of an animation goes on instead of starting from the seed."""
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _scene(rtlib, res):
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=5, seed=2, res=res)
    cam = scenes.look_at_camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, res, res)
    ctx = rtlib.Context(0)
    return ctx, rtlib.Scene(ctx, scene), dict(frame, camera=cam, lights=[dict(frame["lights"][0], r=0.6)])


@pytest.mark.parametrize("start", [0, 12345])
def test_nothing_runs_after_the_call(rtlib, start):
    """Frames of tens of thousands of refills (0.1 us each): read ahead for a next
    frame whole, the device is busy for milliseconds more."""
    ctx, sc, frame = _scene(rtlib, 720)
    p, left = start, []
    for _ in range(6):
        r = sc.render_soft(frame, 64, stream_offset=p)
        t = time.perf_counter()
        torch.cuda.synchronize()
        left.append(time.perf_counter() - t)
        assert r["stream_end"] - p > 624 * 50000
        p = r["stream_end"]
    assert sorted(left)[3] < 1.0e-3, left
    ctx.close()


@pytest.mark.parametrize("res,samples", [(9, 1), (14, 2), (11, 3), (9, 5)])
def test_animation_goes_on(rtlib, res, samples):
    """Small frames (150 to 770 numbers) 100,000 refills into the stream: starting
    from the seed takes 8 ms, a frame 0.2."""
    ctx, sc, frame = _scene(rtlib, res)
    p = 624 * 100000
    p = sc.render_soft(frame, samples, stream_offset=p)["stream_end"]
    slow = 0
    for _ in range(60):
        t = time.perf_counter()
        p = sc.render_soft(frame, samples, stream_offset=p)["stream_end"]
        slow += time.perf_counter() - t > 4.0e-3
    assert slow < 2
    ctx.close()
