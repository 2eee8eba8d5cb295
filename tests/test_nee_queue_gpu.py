"""The queued visibility rays of PathTracerTest (k_shade -> k_extend_p / k_shadow): a scene
rendered alone, in a batch beside plain and guided scenes and in passes of other sizes gives
the same samples, so the films differ by FP64 summation order alone."""
import numpy as np
import pytest

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [0, 1, 6])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 7), (64, 50)])
def test_nee_alone_and_beside_other_scenes(depth, w, h):
    sc = [scenes.material_spheres(w, h), scenes.medium_scene(w, h), scenes.cornell_box(w, h)]
    ctxs = []
    for s in sc:
        c = rx.Context(0)
        c.set_scene(s)
        c.build_accel()
        ctxs.append(c)
    ctxs[2].guide_init(seed=2, box=((0, 0, 0), (5.56, 5.56, 5.56)), train_passes=0, steps_per_pass=0)
    opt = [dict(spp=5, max_depth=depth, nee=True, seed=3), dict(spp=4, max_depth=depth + 1, nee=True, rr_mode=1, seed=4),
           dict(spp=3, max_depth=depth, seed=5)]
    alone = [c.render_pt(s.camera, **o)[0] for c, s, o in zip(ctxs, sc, opt)]
    small, _, st = ctxs[0].render_pt(sc[0].camera, paths_per_pass=17 if w < 64 else 5000, **opt[0])
    np.testing.assert_allclose(small, alone[0], rtol=1e-9, atol=1e-15)
    assert st["shadow_rays"] > 0 or depth == 0 or w == 1
    for graph in (False, True):
        for guided in (False, True):
            items = [(c, s.camera, dict(o, guided=guided and k == 2)) for k, (c, s, o) in enumerate(zip(ctxs, sc, opt))]
            films, _ = ctxs[0].render_pt_batch(items, use_graph=graph, paths_per_pass=4096)
            for k in (0, 1) if guided else (0, 1, 2):
                np.testing.assert_allclose(films[k], alone[k], rtol=1e-9, atol=1e-15)
            assert np.isfinite(films[2]).all()
    for c in ctxs:
        c.close()
