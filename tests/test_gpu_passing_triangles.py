"""Any-hit rays pass light and transparent triangles; scenes that have some
give those rays a copy of the nodes without the children that hold nothing
else.  The answers are those of a scene of the other triangles alone, after a
build, a refit and a rebuild, with none, one, some, most and all triangles
passed, spread over the scene or in one part of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def heights(scene, k):
    v = scene["verts"].copy()
    v[:, 1] += (20.0 * np.sin(0.013 * k * v[:, 0]) * np.cos(0.009 * v[:, 2])).astype(np.float32)
    return v


@pytest.mark.parametrize("passed", ["none", "one", "some", "most", "part", "all but one", "all"])
@pytest.mark.parametrize("n", [1, 2, 64])
def test_answers_are_the_other_triangles(rtlib, ctx, passed, n):
    from raptor_gb300 import scenes
    scene, _ = scenes.terrain_scene(size_pow2=max(n, 2) if n > 1 else 2)
    scene = dict(scene, tris=scene["tris"][:1] if n == 1 else scene["tris"], mat_of_tri=None)
    nt = len(scene["tris"])
    rng = np.random.default_rng(nt)
    mask = {"none": np.zeros(nt, bool), "one": np.arange(nt) == nt // 2, "some": rng.random(nt) < 0.3,
            "most": rng.random(nt) < 0.97, "part": np.arange(nt) < nt // 2, "all but one": np.arange(nt) != nt // 3,
            "all": np.ones(nt, bool)}[passed]
    flags = np.where(mask, rng.integers(1, 4, nt), 0).astype(np.uint32)
    m = 20000
    lo, hi = scene["verts"].min(0), scene["verts"].max(0)
    o = rng.uniform(lo, hi, (m, 3)).astype(np.float32)
    o[:, 1] = hi[1] + 50.0
    to = rng.uniform(lo, hi, (m, 3)).astype(np.float32)
    to[:, 1] = lo[1] - 50.0
    d = to - o
    dist = np.linalg.norm(d, axis=1).astype(np.float32)
    rays = rtlib.rays_array(o, d / dist[:, None], dist)
    sc = rtlib.Scene(ctx, dict(scene, flags=flags))
    closest = sc.closest(rays)
    for step in range(3):
        if step == 1:
            sc.refit_vertices(heights(scene, 1))
        if step == 2:
            sc.update_vertices(heights(scene, 2))
        got = np.asarray(sc.any(rays))
        keep = ~mask
        if keep.any():
            other = rtlib.Scene(ctx, {"verts": heights(scene, step) if step else scene["verts"],
                                      "tris": scene["tris"][keep], "vattr": None,
                                      "flags": np.zeros(int(keep.sum()), np.uint32)})
            assert np.array_equal(got, np.asarray(other.any(rays)))
            other.close()
        else:
            assert not got.any()
    # closest hits still meet every triangle
    sc.update_vertices(scene["verts"])
    again = sc.closest(rays)
    assert np.array_equal(np.asarray(closest), np.asarray(again))
    sc.close()
