"""Soft-shadow frames trace the rays of a warp's hits 32 at a time in the hits'
order: at sample counts that split a hit's rays over passes and at sizes that
leave lanes without hits, the float frame equals the oracle's, bit for bit, on
99.9 % of the pixels with the same primary hit (ties at edges), and the stream
ends where the oracle's does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (9, 5), (40, 30)], ids=str)
@pytest.mark.parametrize("samples", [2, 3, 31, 32, 33, 64])
def test_hit_rays_match_oracle(rtlib, ctx, oracle, size, samples):
    from raptor_gb300 import scenes
    scene, frame = scenes.glass_scene(freq=6, res=8)
    cam = scenes.look_at_camera((0.3, 0.8, 4.0), (0.0, -0.2, 0.0), 50.0, *size, background=(110.0, 160.0, 230.0))
    mats = [dict(m, rf=0.0, tran=0.0) for m in frame["materials"]]
    frame = dict(frame, camera=cam, materials=mats, lights=[dict(frame["lights"][0], r=0.7), frame["lights"][1]])
    sc = rtlib.Scene(ctx, scene)
    out = sc.render_soft(frame, samples, stream_offset=99, want_float=True)
    ref = oracle.OracleScene(scene).render_soft(frame, samples, stream_offset=99, want_ids=True, want_float=True)
    same = sc.render(dict(frame, lights=[], materials=None), want_ids=True)["ids"] == ref["ids"]
    sc.close()
    assert same.all() and out["stream_end"] == ref["stream_end"]
    exact = (out["fimg"].view(np.uint32) == ref["fimg"].view(np.uint32)).all(-1)
    assert exact.mean() > 0.999, exact.mean()
