"""Contexts that render one after another share the device memory their renders keep, it is given
back on request and with the last context, and a render after that gives the same film."""
import gc

import numpy as np
import pytest
import torch

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_contexts_share_the_memory_their_renders_keep():
    gc.collect()  # contexts that earlier tests have dropped
    sc = scenes.cornell_box(1024, 1024)
    with rx.Context(0) as c:  # modules and the like are loaded
        c.set_scene(sc)
        c.build_accel()
        c.render_pt(sc.camera, 1)
        c.release_memory()
        start = _free()
    ctxs, free, films = [], [], []
    for k in range(6):
        c = rx.Context(0)
        c.set_scene(sc)
        c.build_accel()
        films.append(c.render_pt(sc.camera, 4, max_depth=6, seed=3)[0])  # 2^22 paths, 184 bytes each
        ctxs.append(c)
        free.append(_free())
    need = 184 << 22
    assert start - free[0] >= need  # the first context's render keeps its buffers
    assert free[0] - free[5] < need // 4  # five more contexts of 36 triangles, and no more buffers
    ctxs[2].release_memory()
    assert _free() - free[5] >= need
    films.append(ctxs[4].render_pt(sc.camera, 4, max_depth=6, seed=3)[0])
    for f in films[1:]:  # the FP64 film's order of summation differs
        np.testing.assert_allclose(f, films[0], rtol=1e-12, atol=1e-15)
    for c in ctxs:
        c.close()
    assert _free() >= start - 64 * MB
