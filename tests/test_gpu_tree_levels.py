"""Distributed frames on per-pixel streams trace the ray trees of all pixels a
level at a time: frames that leave warps partly without rays, sets of many, few
and single rays, several lights a hit, and trees too large for the pool of
nodes (their subtrees are walked one by one) equal the oracle's frames, which
draw the same numbers, as closely as the other per-pixel-stream frames do: bit
for bit on 99.9 % of the pixels with the same primary hit (ties at edges)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NTHREADS = max(1, os.cpu_count() or 1)


def compare(rtlib, ctx, oracle, scene, frame, soft, diffuse, seed=5):
    sc = rtlib.Scene(ctx, scene)
    out = sc.render_distributed(frame, soft=soft, diffuse=diffuse, stream=rtlib.RT_STREAM_PIXEL, seed=seed,
                                want_float=True)
    assert out["stats"].status == 0
    ref = oracle.OracleScene(scene).render_distributed(frame, soft=soft, diffuse=diffuse, stream=oracle.STREAM_PIXEL,
                                                       seed=seed, threads=NTHREADS, want_ids=True, want_float=True)
    same = sc.render(dict(frame, lights=[], materials=None), want_ids=True)["ids"] == ref["ids"]
    exact = (out["fimg"].view(np.uint32) == ref["fimg"].view(np.uint32)).all(-1)
    again = sc.render_distributed(frame, soft=soft, diffuse=diffuse, stream=rtlib.RT_STREAM_PIXEL, seed=seed,
                                  want_float=True)
    assert np.array_equal(again["fimg"].view(np.uint32), out["fimg"].view(np.uint32))
    sc.close()
    assert same.mean() > 0.99 and exact[same].mean() > 0.999, (same.mean(), exact[same].mean())
    assert abs(out["stream_end"] - ref["drawn"]) <= 0.001 * max(ref["drawn"], 1000)
    return out


@pytest.mark.parametrize("size", [(1, 1), (5, 7), (33, 31), (64, 48)], ids=str)
@pytest.mark.parametrize("soft,diffuse", [(1, 0), (4, 1), (3, 5), (16, 16)])
def test_levels_match_oracle(rtlib, ctx, oracle, size, soft, diffuse):
    from raptor_gb300 import scenes
    scene, frame = scenes.glass_scene(freq=6, res=8)
    cam = scenes.look_at_camera((0.3, 0.8, 4.0), (0.0, -0.2, 0.0), 50.0, *size, background=(110.0, 160.0, 230.0))
    mats = [dict(frame["materials"][0], rfd=0.05, td=0.0), dict(frame["materials"][1], rfd=0.02, td=0.03)]
    lights = [dict(frame["lights"][0], r=0.7), frame["lights"][1]]
    compare(rtlib, ctx, oracle, scene, dict(frame, camera=cam, materials=mats, lights=lights), soft, diffuse)


@pytest.mark.parametrize("diffuse", [8, 48])
def test_trees_beyond_the_pool(rtlib, ctx, oracle, diffuse):
    """Inside a closed box every ray hits and every hit of power above the
    limit has a whole set: with 48 rays a camera ray has 48 + 576 nodes below
    it, more than the pool holds for each item."""
    from raptor_gb300 import scenes
    scene, frame = scenes.glass_scene(freq=2, res=8)
    v = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32) * 3.0
    q = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    t = np.array([w for a, b, c, d in q for w in ((a, b, c), (a, c, d))], np.int32)
    box = {"verts": v, "tris": t, "vattr": None, "flags": np.zeros(len(t), np.uint32),
           "mat_of_tri": np.zeros(len(t), np.int32)}
    cam = scenes.look_at_camera((0.3, 0.8, 1.5), (0.1, -0.2, 0.0), 70.0, 40, 24, background=(1.0, 2.0, 3.0))
    mats = [dict(frame["materials"][0], rf=0.4, rfd=0.2, td=0.0)]
    lights = [dict(frame["lights"][0], pos=(0.5, 0.7, 0.2), r=0.3)]
    out = compare(rtlib, ctx, oracle, box, dict(frame, camera=cam, materials=mats, lights=lights), 2, diffuse)
    below = diffuse * (1 + diffuse // 4)
    assert out["stats"].secondary_rays >= 0.99 * 40 * 24 * below
