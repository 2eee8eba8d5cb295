"""k_shade takes each block's paths by material: films at path counts around its block sizes
(256 without media, 512 with) equal the ones of many small passes, whose blocks hold other
paths, up to FP64 summation order."""
import numpy as np
import pytest

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nee", [False, True])
@pytest.mark.parametrize("scene", ["spheres", "medium"])
def test_films_do_not_depend_on_the_blocks(scene, nee):
    sc = scenes.material_spheres(64, 64) if scene == "spheres" else scenes.medium_scene(64, 64)
    with rx.Context(0) as ctx:
        ctx.set_scene(sc)
        ctx.build_accel()
        for w, h, spp in ((1, 1, 1), (255, 1, 1), (257, 1, 1), (511, 1, 1), (171, 3, 1), (64, 48, 3)):
            cam = scenes.Camera(w, h, max(1, h), sc.camera.position, sc.camera.focus, sc.camera.up)
            one = ctx.render_pt(cam, spp, max_depth=7, nee=nee, seed=w)[0]
            many = ctx.render_pt(cam, spp, max_depth=7, nee=nee, seed=w, paths_per_pass=101)[0]
            np.testing.assert_allclose(one, many, rtol=1e-9, atol=1e-15)


def test_large_frames_run_in_even_passes():
    """Frames beyond one pass of 2^24 paths, and just above 2^22, equal the ones of an explicit
    pass size up to FP64 summation order."""
    sc = scenes.cornell_box(1024, 1024)
    with rx.Context(0) as ctx:
        ctx.set_scene(sc)
        ctx.build_accel()
        for w, h, spp in ((2049, 2048, 1), (1024, 1025, 17)):
            cam = scenes.cornell_camera(w, h)
            one, sq, st = ctx.render_pt(cam, spp, max_depth=3, seed=w, want_sq=True)
            many, sq2, st2 = ctx.render_pt(cam, spp, max_depth=3, seed=w, want_sq=True, paths_per_pass=1 << 22)
            assert st["paths"] == st2["paths"] == w * h * spp and st["extension_rays"] == st2["extension_rays"]
            np.testing.assert_allclose(one, many, rtol=1e-9, atol=1e-15)
            np.testing.assert_allclose(sq, sq2, rtol=1e-9, atol=1e-15)
