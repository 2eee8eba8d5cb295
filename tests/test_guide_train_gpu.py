"""The training kernel at the edges of its tiles (128 records, two tiles a CTA), and the sums
it keeps between steps: gradients and Adam steps in any order start from clear ones.

The gradient is a mean over the records, so with equal weights the gradient of 2 m records is
the mean of those of its halves. Halving the count doubles every back-propagated value
exactly, BF16 roundings included, so the two differ by the order of FP32 sums alone (a record
lost or counted twice moves them by about 1 / m)."""
import numpy as np
import pytest
import torch

import renderx_gb300 as rx
from oracle import guide_mlp as gm

pytestmark = pytest.mark.gpu
BOX = ((0.0, 0.0, 0.0), (5.56, 5.56, 5.56))


def _records(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 16), np.float32)
    r[:, 0:3] = rng.random((n, 3)) * 5.56
    for k in (3, 6, 9):
        v = rng.normal(size=(n, 3))
        r[:, k:k + 3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    r[:, 12] = 1.0
    return r


@pytest.mark.parametrize("m", [1, 31, 63, 64, 65, 127, 128, 129, 257, 152 * 128 + 1])
def test_gradient_of_two_halves(m):
    recs = _records(2 * m, m)
    rng = np.random.default_rng(2)
    p = gm.init_params(9)
    p = (p + rng.normal(scale=0.03, size=p.shape).astype(np.float32) * (p != 0)).astype(np.float32)
    with rx.Context(0) as ctx:
        ctx.guide_init(seed=9, box=BOX)
        ctx.guide_set_params(p)
        loss, g = ctx.guide_gradient(recs)
        la, ga = ctx.guide_gradient(recs[:m])
        lb, gb = ctx.guide_gradient(recs[m:])
        stepped = ctx.guide_train_step(torch.from_numpy(recs).cuda(), 2 * m)
        after = ctx.guide_params()
        ctx.guide_set_params(p)
        loss2, g2 = ctx.guide_gradient(recs)
    scale = max(1.0, abs(loss))
    assert np.linalg.norm(g) > 0
    assert np.linalg.norm(g - 0.5 * (ga + gb)) <= 5e-5 * np.linalg.norm(g)
    assert abs(loss - 0.5 * (la + lb)) <= 1e-5 * scale
    assert np.linalg.norm(g2 - g) <= 5e-5 * np.linalg.norm(g)
    assert abs(loss2 - loss) <= 1e-5 * scale and abs(stepped - loss) <= 1e-5 * scale
    assert np.abs(after - p).max() <= 5.1e-3  # Adam's first step: at most its step size


@pytest.mark.parametrize("n", [128, 5000])
def test_captured_steps(n):
    """Steps in a replayed CUDA graph do what steps launched one by one do: the same loss after
    twelve. Float atomics move single weights of undecided gradient sign by up to a step, which
    the loss does not see to first order (5e-3 of it allowed)."""
    recs = _records(n, n)
    dev = torch.from_numpy(recs).cuda()
    p = gm.init_params(9)
    with rx.Context(0) as ctx:
        ctx.guide_init(seed=9, box=BOX)
        losses = []
        for captured in (False, True):
            s = torch.cuda.Stream()
            # not captured: the batch's descriptor goes to the device with its first step
            ctx.guide_train_step(dev, n, stream=s.cuda_stream)
            ctx.guide_set_params(p)
            torch.cuda.synchronize()
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=s):
                    for _ in range(4):
                        ctx.guide_train_step(dev, n, stream=s.cuda_stream, want_loss=False)
                for _ in range(3):
                    graph.replay()
            else:
                for _ in range(12):
                    ctx.guide_train_step(dev, n, stream=s.cuda_stream, want_loss=False)
            torch.cuda.synchronize()
            moved = np.abs(ctx.guide_params() - p)
            assert moved.max() > 0.02  # a weight whose gradient keeps its sign: 12 steps of 5e-3
            losses.append(ctx.guide_gradient(recs)[0])
    assert abs(losses[1] - losses[0]) <= 5e-3 * max(1.0, abs(losses[0]))
