"""A build clears its words, bounds and segment range in one launch and reads
them back in one copy: hierarchies of few, odd and no triangles, one after
another on one context with every builder, and batches with empty scenes between
others, answer as the oracle does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("builder", [0, 1, 2])
def test_builds_in_turn(rtlib, oracle, builder):
    from raptor_gb300 import scenes
    ctx = rtlib.Context(0)
    ctx.set_option(rtlib.RT_OPT_BUILDER, builder)
    full, _ = scenes.icosphere_scene(freq=8, res=8)
    rng = np.random.default_rng(2)
    o = rng.normal(size=(500, 3))
    o = (3.0 * o / np.linalg.norm(o, axis=1)[:, None]).astype(np.float32)
    d = rng.uniform(-0.8, 0.8, (500, 3)).astype(np.float32) - o
    d = (d / np.linalg.norm(d, axis=1)[:, None]).astype(np.float32)
    for n in (1, 2, 3, 17, 129, 641, 1280, 5):
        n = min(n, len(full["tris"]))
        scene = dict(full, tris=np.ascontiguousarray(full["tris"][:n]), flags=None, mat_of_tri=None)
        sc = rtlib.Scene(ctx, scene)
        got = sc.closest(rtlib.rays_array(o, d, np.full(500, 3e38, np.float32)))
        ids, t, _, _ = oracle.OracleScene(dict(scene, flags=np.zeros(n, np.uint32))).closest(o, d)
        hit = ids >= 0
        assert np.array_equal(np.asarray(got)["tri"] >= 0, hit)
        assert np.array_equal(np.asarray(got)["t"][hit], t[hit])
        sc.close()
    ctx.close()


def test_batch_with_empty_scenes(rtlib, ctx):
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=4, res=8)
    frame = dict(frame, camera=scenes.look_at_camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, 24, 16))
    empty = dict(scene, tris=np.zeros((0, 3), np.int32), flags=np.zeros(0, np.uint32))
    want = {}
    for key, s in (("full", scene), ("empty", empty)):
        sc = rtlib.Scene(ctx, s)
        want[key] = sc.render(frame)["rgb"]
        sc.close()
    b = rtlib.Batch(ctx)
    order = ["empty", "full", "empty", "full", "full"]
    idx = [b.add_scene(scene if k == "full" else empty) for k in order]
    for _ in range(2):
        b.build()
        out = [torch.zeros((16, 24, 3), dtype=torch.uint8, device="cuda") for _ in order]
        torch.cuda.synchronize()
        b.set_jobs([rtlib.make_job(i, frame, r) for i, r in zip(idx, out)])
        b.render()
        for k, r in zip(order, out):
            assert np.array_equal(r.cpu().numpy(), want[k])
    b.close()
