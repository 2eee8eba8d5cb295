"""Batches small enough for the one-launch closest hit (k_trace_once), at the sizes where its
split over warps changes and at its upper limit, against the persistent walk with its
separate check and re-walk kernels (bit for bit) and the CPU oracle."""
import numpy as np
import pytest
import torch

import oracle
import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


def _rays(n, seed):
    o, d = scenes.hit_rays(n, seed=seed)
    d[:: 7, 1] = 0.0  # some directions with a zero component, some rays that leave the scene
    o[:: 11] += 40.0
    return rx.rays_to_array(o, d)


@pytest.mark.parametrize("spheres,subdiv", [(0, 0), (6, 3)])
def test_once_matches_persistent_walk(spheres, subdiv):
    sc = scenes.sphere_field(spheres, subdiv, seed=2) if spheres else scenes.cornell_box()
    f = sc.flatten()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w = 16 * sms
    with rx.Context(0) as ctx:
        ctx.set_scene(sc)
        ctx.build_accel()
        for n in (1, 2, 31, 33, w - 1, w, w + 1, 2 * w + 1, 16 * w + 5, 32 * w - 1, 1024 * sms, 1024 * sms + 1):
            r = _rays(n, n)
            d = torch.from_numpy(r).cuda()
            out = []
            for variant in (4, 3):
                ctx.set_trace_config(variant, 12)
                tid = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
                dist = torch.full((n + 1,), -7.0, device="cuda")
                ctx.trace_closest_device(d, n, tid, dist, stream=torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                assert int(tid[n]) == -7 and float(dist[n]) == -7.0
                out.append((tid[:n].cpu().numpy(), dist[:n].cpu().numpy()))
            assert np.array_equal(out[0][0], out[1][0]), n
            assert np.array_equal(out[0][1].view(np.int32), out[1][1].view(np.int32)), n
            if n <= 33:
                t, s = oracle.RefTree(f["verts"], f["tris"]).trace(r[:, 0:3].copy(), r[:, 4:7].copy())
                assert np.array_equal(out[0][0], t) and np.array_equal(out[0][1].view(np.int32), s.view(np.int32))
