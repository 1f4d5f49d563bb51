"""The specular power of whole exponents up to 128 is formed in pairs of floats,
others by the double power (exact frames) or powf with a second shading (byte
frames): frames of both kinds of exponents, at the edges between them, equal the
oracle's, which takes the double power: float frames bit for bit and byte frames
byte for byte on 99.9 % of the pixels with the same primary hit (ties at edges)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [0.0, 0.5, 1.0, 2.0, 3.0, 12.5, 20.0, 63.0, 64.0, 127.0, 128.0, 129.0, 1000.0])
@pytest.mark.parametrize("ks", [64.0, 255.0])
def test_frames_match_oracle(rtlib, ctx, oracle, ns, ks):
    from raptor_gb300 import scenes
    scene, frame = scenes.icosphere_scene(freq=12, seed=5, res=8)
    cam = scenes.look_at_camera((0.0, 0.5, 3.0), (0.0, 0.0, 0.0), 50.0, 120, 90, background=(1.0, 2.0, 3.0))
    lights = [scenes.point_light((1.0, 2.0, 5.0)), scenes.point_light((-4.0, 1.0, 3.0), rgb=(90.0, 200.0, 30.0))]
    material = dict(frame["material"], ns=ns, ks=(ks, ks, 0.5 * ks))
    frame = dict(frame, camera=cam, lights=lights, material=material, materials=[material])
    scene = dict(scene, mat_of_tri=None)
    sc = rtlib.Scene(ctx, scene)
    flt = sc.render_soft(frame, 1, want_float=True)
    byte = sc.render(dict(frame, materials=None), want_ids=True)
    sc.close()
    ref = oracle.OracleScene(scene).render_soft(frame, 1, want_ids=True, want_float=True)
    same = byte["ids"] == ref["ids"]
    assert same.mean() > 0.99
    exact = (flt["fimg"].view(np.uint32) == ref["fimg"].view(np.uint32)).all(-1)
    assert exact[same].mean() > 0.999, exact[same].mean()
    assert (byte["rgb"] == ref["rgb"]).all(-1)[same].mean() > 0.999
