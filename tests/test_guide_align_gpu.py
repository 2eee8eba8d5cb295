"""rx_guide_eval_device writes its raw outputs by 16-byte copies: an output pointer that is not
16-byte aligned is refused before anything is launched."""
import numpy as np
import pytest
import torch

import renderx_gb300 as rx

pytestmark = pytest.mark.gpu


def test_misaligned_outputs_are_refused():
    n = 300
    recs = torch.rand(n, 16, device="cuda")
    raw = torch.full((40 * n + 4,), -9.0, device="cuda")
    pdf = torch.full((n + 1,), -9.0, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    with rx.Context(0) as ctx:
        ctx.guide_init(seed=5, box=((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)))
        for k in (1, 2, 3):
            with pytest.raises(rx.RxError, match="16-byte aligned"):
                ctx.guide_eval_device(recs, n, raw[k:], pdf, stream=stream)
        torch.cuda.synchronize()
        assert bool((raw == -9.0).all()) and bool((pdf == -9.0).all())
        # aligned rows, and densities at any float's alignment
        ctx.guide_eval_device(recs, n, raw[4:], pdf[1:], stream=stream)
        torch.cuda.synchronize()
        want, q = ctx.guide_eval(recs.cpu().numpy())
    assert np.array_equal(raw[4:].cpu().numpy().reshape(n, 40), want) and np.array_equal(pdf[1:].cpu().numpy(), q)
    assert bool((raw[:4] == -9.0).all()) and float(pdf[0]) == -9.0
