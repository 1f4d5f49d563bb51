"""Anti-aliased frames whose specular exponent is not whole queue the pixels that
land near a truncation and shade them again exactly, in step or one by one by how
many they are.  Either way the frame is the downsampled exact float image, byte
for byte: queues of no, a few hundred and tens of thousands of pixels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(7, 5), (96, 64), (640, 480), (1920, 1200)])
@pytest.mark.parametrize("aa", [(2, 2), (1, 3)])
def test_frame_is_the_exact_image(rtlib, oracle, size, aa):
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=9, seed=4)
    cam = scenes.look_at_camera((0.0, 0.5, 4.0), (0.0, 0.0, 0.0), 60.0, *size)
    frame = dict(frame, camera=cam, material=dict(frame["material"], ns=20.5))
    ctx = rtlib.Context(0)
    sc = rtlib.Scene(ctx, scene)
    fimg = sc.render_image(frame, aa=aa)["fimg"]
    rgb = sc.render_aa(frame, *aa)["rgb"]
    assert np.array_equal(rgb, oracle.downsample_rgb8(fimg, *aa))
    ctx.close()
