"""The inference kernel at the edges of its tiles (128 rows), warps (32), and spread over SMs:
a batch's rows are independent, so a prefix of any length gives the same bits, and nothing
beyond it is written. The density against the oracle's mixture of the same raw outputs, with
test_guide_gpu.py's tolerance."""
import numpy as np
import pytest
import torch

import renderx_gb300 as rx
from oracle import guide_mlp as gm

pytestmark = pytest.mark.gpu
BOX = ((0.0, 0.0, 0.0), (5.56, 5.56, 5.56))


def test_rows_do_not_depend_on_the_batch():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    big = sms * 1024 + 333
    g = torch.Generator(device="cuda").manual_seed(4)
    recs = torch.rand(big, 16, generator=g, device="cuda") * 5.56
    for k in (3, 6, 9):
        v = torch.randn(big, 3, generator=g, device="cuda")
        recs[:, k:k + 3] = v / v.norm(dim=1, keepdim=True)
    stream = torch.cuda.current_stream().cuda_stream
    with rx.Context(0) as ctx:
        ctx.guide_init(seed=5, box=BOX)
        p = gm.init_params(5)
        ctx.guide_set_params((p + np.random.default_rng(1).normal(scale=0.1, size=p.shape) * (p != 0)).astype(np.float32))

        def run(n, raw=True, pdf=True):
            o = torch.full((n + 1, 40), -9.0, device="cuda") if raw else None
            q = torch.full((n + 1,), -9.0, device="cuda") if pdf else None
            ctx.guide_eval_device(recs, n, o, q, stream=stream)
            torch.cuda.synchronize()
            for x in (o, q):
                assert x is None or bool((x[n] == -9.0).all())
            return None if o is None else o[:n], None if q is None else q[:n]

        raw, pdf = run(big)
        for n in (1, 31, 33, 127, 128, 129, 1023, 1025, 128 * sms - 1, 128 * sms, 128 * sms + 1, 1024 * sms, 1024 * sms + 1):
            o, q = run(n)
            assert torch.equal(o, raw[:n]) and torch.equal(q, pdf[:n]), n
        assert torch.equal(run(777, pdf=False)[0], raw[:777]) and torch.equal(run(777, raw=False)[1], pdf[:777])
    k = slice(0, 4000)
    want = gm.mixture_pdf(raw[k].cpu().numpy().astype(np.float64), recs[k, 9:12].cpu().numpy())
    assert np.allclose(pdf[k].cpu().numpy(), want, rtol=1e-3, atol=1e-6)
