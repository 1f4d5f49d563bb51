"""Small ray queries run in one pass with fewer rays to a warp, host rays
through pinned memory: their answers equal, bit for bit, those of the same
rays inside a large query (which takes the work-queue kernel), at every
boundary of the dispatch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TOTAL = 400000


@pytest.fixture(scope="module")
def setup(rtlib):
    from raptor_gb300 import scenes
    scene, _ = scenes.terrain_scene(size_pow2=64)
    c = rtlib.Context(0)
    sc = rtlib.Scene(c, scene)
    rng = np.random.default_rng(8)
    lo, hi = scene["verts"].min(0), scene["verts"].max(0)
    o = rng.uniform(lo, hi, (TOTAL, 3)).astype(np.float32)
    o[:, 1] = hi[1] + 5.0
    d = (rng.uniform(lo - 50.0, hi + 50.0, (TOTAL, 3)) - o).astype(np.float32)
    dist = np.linalg.norm(d, axis=1).astype(np.float32)
    rays = rtlib.rays_array(o, d / dist[:, None], dist * rng.uniform(0.5, 1.5, TOTAL).astype(np.float32))
    dev = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
    hits = torch.empty((TOTAL, 4), dtype=torch.int32, device="cuda")
    occ = torch.empty(TOTAL, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    sc.closest_into(dev, hits)
    rtlib._check(rtlib.lib().rt_trace_any(sc.h, rtlib.ptr(dev), TOTAL, rtlib.ptr(occ)))
    hits, occ = hits.cpu().numpy(), occ.cpu().numpy()
    assert 0.2 < (hits[:, 0] >= 0).mean() < 1.0 and 0.05 < occ.mean() < 0.95
    yield sc, rays, dev, hits, occ
    c.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 4863, 4864, 4865, 9729, 16384, 16385, 155647, 155648, 155649])
@pytest.mark.parametrize("where", ["host", "device", "host-to-device", "device-to-host"])
def test_few_rays(rtlib, setup, n, where):
    sc, rays, dev, hits, occ = setup
    k = (TOTAL - n) // 2   # not always from the first ray
    hi = where in ("host", "host-to-device")
    ho = where in ("host", "device-to-host")
    src = np.ascontiguousarray(rays[k:k + n]) if hi else dev[k:k + n]
    h = np.full((n, 4), -7, np.int32) if ho else torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
    a = np.full(n, 9, np.uint8) if ho else torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    lib = rtlib.lib()
    rtlib._check(lib.rt_trace_closest(sc.h, rtlib.ptr(src), n, rtlib.ptr(h)))
    rtlib._check(lib.rt_trace_any(sc.h, rtlib.ptr(src), n, rtlib.ptr(a)))
    h, a = (h, a) if ho else (h.cpu().numpy(), a.cpu().numpy())
    assert np.array_equal(h, hits[k:k + n])
    assert np.array_equal(a, occ[k:k + n])
