"""The reference's random stream on the device: windows of whole refills (624
numbers), read ahead past the frame, carried over, skipped to or restarted
from the seed.  Whatever frames came before, a frame at offset p must draw
numbers p, p + 1, ...: each frame of a sequence on one context equals the same
frame on a context of its own, bytes and stream position."""
import pytest

pytestmark = pytest.mark.gpu

SEQUENCES = {
    "edges": [0, 1, 623, 624, 625, 1247, 1248],
    "repeat": [5000, 5000, 5000],
    "back": [70000, 624, 69999, 0],
    "ahead": [0, 10 ** 6, 10 ** 6 + 311, 2 * 10 ** 6],
    "consecutive": [17, None, None, None, None],          # None: where the last frame ended
    "mixed": [0, None, 0, None, 3 * 624, None],
}


@pytest.mark.parametrize("name", sorted(SEQUENCES))
def test_sequence(rtlib, name):
    import numpy as np
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=5, seed=2, res=24)
    c = rtlib.Context(0)
    sc = rtlib.Scene(c, scene)
    end = 0
    for k, p in enumerate(SEQUENCES[name]):
        # frames of different sizes and sample counts draw more and less than the read-ahead
        res, n = ((24, 7), (40, 3), (11, 16))[k % 3]
        cam = scenes.look_at_camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, res, res)
        f = dict(frame, camera=cam, lights=[dict(frame["lights"][0], r=0.6)])
        p = end if p is None else p
        got = sc.render_soft(f, n, stream_offset=p)
        fresh = rtlib.Context(0)
        want = rtlib.Scene(fresh, scene).render_soft(f, n, stream_offset=p)
        assert np.array_equal(got["rgb"], want["rgb"]), (k, p)
        assert got["stream_end"] == want["stream_end"] > p
        end = got["stream_end"]
        fresh.close()
    sc.close()
    c.close()


def test_sequence_matches_restatement(rtlib, oracle):
    """Frames drawn across several refills against the CPU restatement's
    serial generator (the camera's centre column may tie, as in the other
    soft-shadow tests: 99 % of the pixels equal, the position equal)."""
    import numpy as np
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=5, seed=2, res=33)
    frame = dict(frame, lights=[dict(frame["lights"][0], r=0.6)])
    c = rtlib.Context(0)
    sc = rtlib.Scene(c, scene)
    osc = oracle.OracleScene(scene)
    p = 600
    for _ in range(3):
        got = sc.render_soft(frame, 5, stream_offset=p)
        want = osc.render_soft(frame, 5, stream_offset=p)
        assert (got["rgb"] == want["rgb"]).all(-1).mean() >= 0.99
        assert got["stream_end"] == want["stream_end"]
        p = got["stream_end"]
    c.close()
