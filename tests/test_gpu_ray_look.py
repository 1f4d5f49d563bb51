"""The look at the rays of a large any-hit query, and the bound of the host rays
that a closest query stages itself.  Whatever kernel answers, the answers are
those of the same rays in small queries: scattered rays that are through after a
node or two but for some, the share of these on both sides of one in 64 and in
none, some or all of the groups looked at."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("isect", [0, 1])
@pytest.mark.parametrize("share", [0.0, 0.005, 0.03, 1.0])
def test_answers_equal_small_queries(rtlib, isect, share):
    """A sphere on a large ground: rays up from scattered points but for `share`
    of them, which go for the sphere."""
    from raptor_gb300 import scenes
    scene, _ = scenes.icosphere_scene(freq=9, seed=4)
    ctx = rtlib.Context(0)
    ctx.set_option(rtlib.RT_OPT_INTERSECTOR, isect)
    sc = rtlib.Scene(ctx, scene)
    n = 4 * 8 * 128 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    rng = np.random.default_rng(5)
    o = rng.uniform((-20.0, -0.9, -20.0), (20.0, 3.0, 20.0), (n, 3)).astype(np.float32)
    to = o + np.array([0.3, 1.0, 0.2], np.float32)
    near = rng.random(n) < share
    to[near] = rng.uniform(-1.2, 1.2, (int(near.sum()), 3))
    d = to - o
    d /= np.linalg.norm(d, axis=1)[:, None]
    rays = rtlib.rays_array(o, d, np.full(n, 100.0, np.float32))
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
    assert (a == 1).any() and (a == 0).any()
    ctx.close()


@pytest.mark.parametrize("n", [12287, 12288, 12289, 16384, 16385])
def test_host_rays_equal_device_rays(rtlib, n):
    from raptor_gb300 import scenes
    scene, _ = scenes.icosphere_scene(freq=9, seed=4)
    ctx = rtlib.Context(0)
    sc = rtlib.Scene(ctx, scene)
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1)[:, None]
    rays = rtlib.rays_array(np.float32([0.0, 2.0, 0.5]) + np.zeros_like(d), d, np.full(n, 5.0, np.float32))
    dev = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
    out = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    sc.closest_into(dev, out)
    rtlib._check(rtlib.lib().rt_trace_any(sc.h, rtlib.ptr(dev), n, rtlib.ptr(occ)))
    assert np.array_equal(sc.closest(rays).view(np.int32).reshape(-1, 4), out.cpu().numpy())
    assert np.array_equal(sc.any(rays), occ.cpu().numpy())
    ctx.close()
