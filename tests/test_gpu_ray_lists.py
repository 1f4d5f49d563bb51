"""Large any-hit queries whose rays start all over the scene let a lane take
another ray when its own is finished.  Their answers equal, byte for byte, those
of the same rays in small queries, at the boundary of the dispatch and past it,
for scattered rays, rays of one point, and lists that are partly either, with
rays that miss everything and rays without a direction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def make_rays(rtlib, scene, n, kind):
    rng = np.random.default_rng(n)
    lo, hi = scene["verts"].min(0), scene["verts"].max(0)
    ext = hi - lo
    o = (lo + ext * rng.uniform(-0.2, 1.2, (n, 3))).astype(np.float32)
    o[:, 1] = hi[1] + ext[1] * rng.uniform(0.05, 0.5, n)
    to = (lo + ext * rng.uniform(-0.1, 1.1, (n, 3))).astype(np.float32)
    if kind == "point":
        o[:] = o[0]
    if kind == "half":
        o[:n // 2] = o[0]
    if kind == "parallel":
        to = o - np.array([0.3, 1.0, 0.2], np.float32) * ext.max()
    d = to - o
    dist = np.linalg.norm(d, axis=1).astype(np.float32)
    d = d / dist[:, None]
    if kind == "odd":
        d[::977] = 0.0
        d[5::977] = (0.0, 1.0, 0.0)
    return rtlib.rays_array(o, d, dist * rng.uniform(0.2, 1.5, n).astype(np.float32))


@pytest.mark.parametrize("isect", [0, 1])
@pytest.mark.parametrize("kind", ["scattered", "point", "half", "parallel", "odd"])
@pytest.mark.parametrize("over", [-1, 0, 1, 77777])
def test_answers_equal_small_queries(rtlib, isect, kind, over):
    from raptor_gb300 import scenes
    scene, _ = scenes.terrain_scene(size_pow2=32)
    flags = np.where(np.random.default_rng(1).random(len(scene["tris"])) < 0.3, 2, 0).astype(np.uint32)
    ctx = rtlib.Context(0)
    ctx.set_option(rtlib.RT_OPT_INTERSECTOR, isect)
    sc = rtlib.Scene(ctx, dict(scene, flags=flags))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 4 * 8 * 128 * sms + over
    rays = make_rays(rtlib, scene, n, kind)
    dev = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
    a = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    b = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rtlib._check(rtlib.lib().rt_trace_any(sc.h, rtlib.ptr(dev), n, rtlib.ptr(a)))
    for k in range(0, n, 100000):
        m = min(100000, n - k)
        rtlib._check(rtlib.lib().rt_trace_any(sc.h, rtlib.ptr(dev[k:k + m]), m, rtlib.ptr(b[k:k + m])))
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert np.array_equal(a, b)
    assert 0.01 < a.mean() < 0.99
    ctx.close()
