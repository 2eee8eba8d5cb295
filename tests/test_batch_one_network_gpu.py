"""A batch in which one network guides: beside plain scenes, or shared by two items of one
context. (The grouped inference of a batch of several scenes needs its sort buffers with one
network as with many.)"""
import numpy as np
import pytest

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", [False, True])
def test_one_network_beside_plain_scenes(shared):
    sc = scenes.cornell_box(40, 30)
    with rx.Context(0) as a, rx.Context(0) as b:
        for c in (a, b):
            c.set_scene(sc)
            c.build_accel()
        a.guide_init(seed=2, box=((0, 0, 0), (5.56, 5.56, 5.56)), train_passes=0, steps_per_pass=0)
        plain = dict(spp=4, max_depth=6, seed=3)
        guided = dict(spp=4, max_depth=6, seed=4, guided=True)
        alone = b.render_pt(sc.camera, **plain)[0]
        items = [(b, sc.camera, plain), (a, sc.camera, guided)] + [(a, sc.camera, dict(guided, seed=5))] * shared
        films, _ = a.render_pt_batch(items)
        np.testing.assert_allclose(films[0], alone, rtol=1e-9, atol=1e-15)
        for f in films[1:]:
            assert np.isfinite(f).all() and f.mean() > 0
