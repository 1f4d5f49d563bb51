"""Frames trace a warp's rays in step, batches ray by ray: the same frame
through either kernel is the same bytes and ids, at sizes that leave warps
partly or wholly without pixels, with no, one and two lights, and with tiles
in which no, some and all rays hit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (8, 4), (9, 5), (33, 2), (65, 31)], ids=str)
@pytest.mark.parametrize("lights", [0, 1, 2])
@pytest.mark.parametrize("which", ["sphere", "terrain"])
def test_frame_equals_batched_frame(rtlib, ctx, size, lights, which):
    from raptor_gb300 import scenes
    if which == "sphere":
        scene, frame = scenes.icosphere_scene(freq=12, seed=3, res=8)
        eye, at = (0.0, 0.5, 4.0), (0.0, 0.0, 0.0)
    else:
        scene, frame = scenes.terrain_scene(size_pow2=64, xres=8, yres=8)
        eye, at = (0.0, 300.0, 0.0), (512.0, 100.0, 512.0)
    cam = scenes.look_at_camera(eye, at, 60.0, *size, background=(10.0, 20.0, 30.0))
    ls = [frame["lights"][0], scenes.point_light((30.0, 400.0, 20.0), rgb=(90.0, 80.0, 70.0))][:lights]
    frame = dict(frame, camera=cam, lights=ls)
    sc = rtlib.Scene(ctx, scene)
    out = sc.render(frame, want_ids=True)
    b = rtlib.Batch(ctx)
    i = b.add_scene(scene)
    b.build()
    rgb = torch.empty((size[1], size[0], 3), dtype=torch.uint8, device="cuda")
    ids = torch.empty((size[1], size[0]), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    b.set_jobs([rtlib.make_job(i, frame, rgb, ids)])
    st = b.render()
    assert np.array_equal(out["rgb"], rgb.cpu().numpy())
    assert np.array_equal(out["ids"], ids.cpu().numpy())
    for k in ("primary_rays", "secondary_rays", "primary_hits"):
        assert getattr(out["stats"], k) == getattr(st, k), k
    b.close()
    sc.close()
