"""Batches just beyond the one-launch closest hit, where the persistent walk's warps wait for all
of their lanes or leave early by the tree's depth and the rays per lane: at both sides of
each limit the answers are those of the walk that always leaves early (variant 3), bit for bit."""
import pytest
import torch

import renderx_gb300 as rx
from renderx_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spheres,subdiv,depth", [(0, 0, (1, 4)), (20, 3, (5, 10)), (50, 4, (11, 14))])
def test_waiting_walk_matches_leaving_walk(spheres, subdiv, depth):
    sc = scenes.sphere_field(spheres, subdiv, seed=1) if spheres else scenes.cornell_box()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lanes = 12 * 128 * sms
    stream = torch.cuda.current_stream().cuda_stream
    with rx.Context(0) as ctx:
        ctx.set_scene(sc)
        ctx.build_accel()
        ctx.set_trace_options(1, 0, 0)  # unbinned
        assert depth[0] <= ctx.stats()["bvh4_depth"] <= depth[1]
        for n in (1024 * sms + 1, lanes - 1, lanes + 1, lanes + lanes // 8, lanes + lanes // 8 + 1, 2 * lanes + 77):
            o, d = scenes.hit_rays(n, seed=n)
            o[:: 11] += 40.0
            rays = torch.from_numpy(rx.rays_to_array(o, d)).cuda()
            out = []
            for variant in (4, 3):
                ctx.set_trace_config(variant, 12)
                tid = torch.full((n,), -7, dtype=torch.int32, device="cuda")
                dist = torch.full((n,), -7.0, device="cuda")
                ctx.trace_closest_device(rays, n, tid, dist, stream=stream)
                out.append((tid, dist.view(torch.int32)))
            assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]), n
            assert int((out[0][0] >= 0).sum()) > n // 2
