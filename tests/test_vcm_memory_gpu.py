"""Device memory of the bidirectional renders: lists whose size varies from iteration to
iteration are not taken anew for each new highest number of connections."""
import gc

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
