"""A batch renders its shadow-ray jobs and its AO jobs in kernels of their own,
side by side: every frame of batches of one kind, of both, in several orders and
launch shapes equals the frame rendered alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(33, 17), (8, 4), (1, 1), (70, 45)]


@pytest.mark.parametrize("kinds", ["L", "A", "LA", "AL", "ALLA", "LLAALAL"])
@pytest.mark.parametrize("config", [dict(), dict(kernel=1, tile_w=16, chunk_tiles=4),
                                    dict(kernel=1, block_threads=256, stack_entries=24), dict(kernel=0)], ids=str)
def test_frames_equal_single_frames(rtlib, ctx, kinds, config):
    from raptor_gb300 import scenes
    b = rtlib.Batch(ctx)
    jobs, want = [], []
    for k, kind in enumerate(kinds):
        scene, frame = scenes.icosphere_scene(freq=5 + k, seed=k, res=8) if k % 2 else scenes.terrain_scene(size_pow2=16)
        eye, at = ((0.0, 0.5, 4.0), (0.0, 0.0, 0.0)) if k % 2 else ((0.0, 300.0, 0.0), (512.0, 100.0, 512.0))
        cam = scenes.look_at_camera(eye, at, 60.0, *SIZES[k % 4], background=(10.0, 20.0, 30.0))
        frame = dict(frame, camera=cam)
        if kind == "A":
            frame = dict(frame, lights=[], ao={"samples": 1 + k, "dist": 1.0 if k % 2 else 80.0, "seed": 40 + k})
        sc = rtlib.Scene(ctx, scene)
        want.append(sc.render(frame, want_ids=True))
        sc.close()
        jobs.append((b.add_scene(scene), frame))
    b.build()
    out = []
    for _, frame in jobs:
        H, W = frame["camera"]["yres"], frame["camera"]["xres"]
        out.append((torch.zeros((H, W, 3), dtype=torch.uint8, device="cuda"),
                    torch.full((H, W), -9, dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    if config:
        b.set_config(**config)
    b.set_jobs([rtlib.make_job(i, f, rgb, ids) for (i, f), (rgb, ids) in zip(jobs, out)])
    for _ in range(2):
        for rgb, ids in out:
            rgb.zero_()
            ids.fill_(-9)
        torch.cuda.synchronize()
        st = b.render()
        for (rgb, ids), w in zip(out, want):
            assert np.array_equal(rgb.cpu().numpy(), w["rgb"])
            assert np.array_equal(ids.cpu().numpy(), w["ids"])
        assert st.primary_rays == sum(w["ids"].size for w in want)
        assert st.secondary_rays == sum(w["stats"].secondary_rays for w in want)
    b.close()
