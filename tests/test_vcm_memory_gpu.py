"""Device memory of the bidirectional renders: lists whose size varies from iteration to
iteration are not taken anew for each new highest number of connections."""
import gc

import numpy as np
import pytest
import torch

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _kept(render):
    """Device bytes that a render leaves with its context (nothing was kept before it)."""
    gc.collect()
    sc = scenes.medium_scene(512, 512)
    with rx.Context(0) as c:
        c.set_scene(sc)
        c.build_accel()
        render(c, scenes.cornell_camera(32, 32))  # modules, streams
        c.release_memory()
        before = _free()
        render(c, sc.camera)
        return before - _free()


@pytest.mark.parametrize("kind", ["bpt", "vcm"])
def test_iterations_do_not_add_memory(kind):
    def run(n):
        if kind == "bpt":
            return lambda c, cam: c.render_bpt(cam, n, max_depth=8, seed=1)
        return lambda c, cam: c.render_vcm(cam, n, 0.01, 0.75, max_depth=8, light_paths=1 << 17, seed=1)
    one, many = _kept(run(1)), _kept(run(60))
    assert one > 100 << 20
    assert many == one


def test_eye_sides_take_a_window():
    # 124 bytes a possible eye vertex (vertices, records, counts and the sorted query list) are
    # kept for the whole image; the queries' eye sides (96 bytes each) for a window of 2^23
    w, h, depth = 2048, 1024, 21
    vertices = w * h * (depth + 3)
    sc = scenes.cornell_box(w, h)
    gc.collect()
    with rx.Context(0) as c:
        c.set_scene(sc)
        c.build_accel()
        c.render_vcm(scenes.cornell_camera(32, 32), 1, 0.01, max_depth=depth, light_paths=64)
        c.release_memory()
        before, during = _free(), []
        c.set_snapshots(1e-6, lambda *a: during.append(_free()))
        c.render_vcm(sc.camera, 1, 0.01, max_depth=depth, light_paths=64)
    used = before - during[0]
    assert 124 * vertices < used < (124 + 96) * vertices


def test_windows_merge_every_query():
    # more queries than a window holds; pair counts equal those of the whole-path loops, and
    # the images with the tolerance of test_merge_matches_full_path_loops
    sc = scenes.cornell_box(2300, 2200)
    with rx.Context(0) as c:
        c.set_scene(sc)
        c.build_accel()
        kw = dict(max_depth=8, light_paths=4096, seed=3)
        fast, sf = c.render_vcm(sc.camera, 1, 0.05, 0.75, **kw)
        full, su = c.render_vcm(sc.camera, 1, 0.05, 0.75, full_path_mis=True, **kw)
    assert sf["merge_queries"] > 1 << 23
    assert sf["merges"] == su["merges"] > 1 << 20
    np.testing.assert_allclose(fast, full, rtol=1e-3, atol=1e-5 * max(full.max(), 1e-3))
