"""Tone mapping of frames with large areas of one value (a sky): pixels of a
warp whose samples are all equal share one entry of the exact redo queue, a
sample equal to the one before it takes its result, and up to 32 samples of a
queued pixel are evaluated by as many lanes.  Against the CPU restatement, as
the other tone-mapped frames: every pixel within one level, 99.9 % equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aa", [(1, 1), (2, 2), (3, 5), (4, 8), (7, 5)], ids=str)
@pytest.mark.parametrize("tone", [{"mode": 5, "gamma": 2.2}, {"mode": 4, "gamma": 1.8, "stretch": True},
                                  {"mode": 6}], ids=lambda t: f"mode{t['mode']}")
def test_flat_areas(rtlib, ctx, oracle, aa, tone):
    from raptor_gb300 import scenes
    W, H = 67, 37
    rng = np.random.default_rng(aa[0] * 10 + aa[1])
    img = np.empty((H * aa[1], W * aa[0], 3), np.float32)
    # bands of one colour each, many of them close to a truncation boundary of
    # some channel for some band; single samples and a block are disturbed
    for r in range(H):
        img[r * aa[1]:(r + 1) * aa[1]] = rng.uniform(5.0, 250.0, 3).astype(np.float32)
    img[:, :W * aa[0] // 5] = rng.uniform(0.0, 300.0, (img.shape[0], W * aa[0] // 5, 3))
    ys, xs = rng.integers(0, img.shape[0], 40), rng.integers(0, img.shape[1], 40)
    img[ys, xs] = rng.uniform(0.0, 255.0, (40, 3))
    cam = scenes.look_at_camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, W, H)
    got = ctx.tone_map_image(img, cam, tone, aa).astype(int)
    want = oracle.downsample_rgb8(oracle.tone_map_frame(img, tone, cam), *aa).astype(int)
    diff = np.abs(got - want).max(-1)
    assert diff.max() <= 1
    assert (diff == 0).mean() >= 0.999
