"""The fused merge kernel (k_merge: walk and pair evaluation in one) against the reference's
loops over each whole joined path, at the sizes where its pair list can go wrong: no photon,
fewer pairs than a warp, lists that several queries share, many pairs per query."""
import numpy as np
import pytest

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["spheres", "medium"])
@pytest.mark.parametrize("w,h,light_paths,radius", [(1, 1, 1, 0.3), (5, 3, 1, 0.5), (7, 9, 33, 0.2), (40, 24, 4096, 0.05),
                                                    (16, 17, 3001, 1.5)])
def test_merge_matches_full_path_loops(scene, w, h, light_paths, radius):
    # the two evaluate the same pairs, so the count is equal and the images differ by FP32
    # rounding (the tolerance of test_factored_mis_matches_full_path_loops)
    sc = scenes.material_spheres(w, h) if scene == "spheres" else scenes.medium_scene(w, h)
    with rx.Context(0) as ctx:
        ctx.set_scene(sc)
        ctx.build_accel()
        for seed in (3, 4):
            kw = dict(max_depth=8, light_paths=light_paths, seed=seed)
            fast, sf = ctx.render_vcm(sc.camera, 2, radius, 0.75, **kw)
            full, su = ctx.render_vcm(sc.camera, 2, radius, 0.75, full_path_mis=True, **kw)
            assert sf["merges"] == su["merges"]
            np.testing.assert_allclose(fast, full, rtol=1e-3, atol=1e-5 * max(full.max(), 1e-3))
