"""The work a user of the library has it do, as cases that can be timed and compared.

A case names a kind of call and its sizes. The kinds are the library's entry points over
the range they are used at: closest-hit batches (device and host buffers, from a handful
of picking rays to the 2^24-ray batch), path-traced frames (one scene, a guided scene,
many small scenes in one wavefront), the guiding network alone (forward pass, training
steps), and the bidirectional estimators. Scenes are the library's seeded synthetic ones;
a case's scene is fixed by its sizes, and the seed makes the rays, records, network
weights and random numbers of the render.

Each case's scene is uploaded and built by prepare(), as a program does once per scene;
run() is one call (or, for training, a few steps) on it.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import renderx_gb300 as rx
from renderx_gb300 import scenes

ROOM = 5.56
BOX = ((0.0, 0.0, 0.0), (ROOM, ROOM, ROOM))
LAYERS = (80, 64, 64, 64, 64)  # input widths of the guiding network's layers, 64 rows each


def listed():
    return [
        # a picking query or one probe's rays: the smallest call, bound by its latency
        dict(name="hit_pick", kind="hit", rays=1000, spheres=0, subdiv=0),
        # a tool's batch over a mid-size scene, device buffers, below the binning size
        dict(name="hit_mid", kind="hit", rays=100_003, spheres=20, subdiv=3),
        # the headline batch: 2^24 rays over 4.1 M triangles, device buffers
        dict(name="hit_large", kind="hit", rays=1 << 24, spheres=200, subdiv=5),
        # a host program's batch from pinned memory, copies both ways included
        dict(name="hit_host", kind="hit_host", rays=3_000_017, spheres=50, subdiv=4),
        # the Cornell box frame: a preview, launch and allocation bound
        dict(name="pt_cornell", kind="pt", spheres=0, subdiv=0, width=256, height=256, spp=16, depth=8, nee=False),
        # a production frame over a million triangles
        dict(name="pt_large", kind="pt", spheres=200, subdiv=4, width=1024, height=1024, spp=16, depth=16, nee=False),
        # many small scenes in one wavefront, half of them light-sampled, some with a medium
        dict(name="pt_batch", kind="batch", items=16, res=128, spp=6, depth=16),
        # a frame sampled through the guiding network
        dict(name="pt_guided", kind="guided", spheres=50, subdiv=3, width=512, height=512, spp=8, depth=12),
        # the guiding network's forward pass on a training-sized query batch
        dict(name="guide_eval", kind="guide_eval", rows=(1 << 20) - 37),
        # a few optimiser steps of the guiding network at its default batch
        dict(name="guide_train", kind="guide_train", rows=1 << 18, steps=4),
        # vertex connection and merging through a medium, a million light paths
        dict(name="vcm_medium", kind="vcm", width=512, height=512, light_paths=1 << 20, iterations=2, depth=16),
        # bidirectional path tracing of the same scene at an odd size
        dict(name="bpt_medium", kind="bpt", width=333, height=251, iterations=2, depth=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _field(rng):
    subdiv = rng.choice([2, 3, 4])
    return dict(spheres=_log(rng, 1, 200 if subdiv < 4 else 100), subdiv=subdiv)


def draw(rng):
    kind = rng.choice(["hit", "hit", "hit_host", "pt", "pt", "batch", "guided", "guide_eval", "guide_train", "vcm", "bpt"])
    if kind == "hit":
        return dict(kind=kind, rays=_log(rng, 500, 1 << 23), **_field(rng))
    if kind == "hit_host":
        return dict(kind=kind, rays=_log(rng, 20_000, 4_000_000), **_field(rng))
    if kind == "pt":
        return dict(kind=kind, **_field(rng), width=_log(rng, 64, 1024), height=_log(rng, 64, 1024),
                    spp=_log(rng, 2, 16), depth=rng.randint(4, 16), nee=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, items=rng.randint(3, 20), res=rng.randint(48, 200), spp=rng.randint(2, 10),
                    depth=rng.randint(6, 16))
    if kind == "guided":
        return dict(kind=kind, **_field(rng), width=_log(rng, 64, 640), height=_log(rng, 64, 640),
                    spp=_log(rng, 2, 12), depth=rng.randint(4, 16))
    if kind == "guide_eval":
        return dict(kind=kind, rows=_log(rng, 1000, 1 << 21))
    if kind == "guide_train":
        return dict(kind=kind, rows=_log(rng, 4096, 1 << 19), steps=rng.randint(1, 4))
    if kind == "vcm":
        return dict(kind=kind, width=_log(rng, 100, 512), height=_log(rng, 100, 512),
                    light_paths=_log(rng, 1 << 14, 1 << 20), iterations=rng.randint(1, 2), depth=rng.randint(8, 16))
    return dict(kind="bpt", width=_log(rng, 64, 512), height=_log(rng, 64, 512), iterations=rng.randint(1, 4),
                depth=rng.randint(8, 16))


# ---- inputs ----------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _scene(spheres: int, subdiv: int):
    """The Cornell box alone, or with a seeded field of displaced icospheres."""
    return scenes.sphere_field(spheres, subdiv, seed=1) if spheres else scenes.cornell_box()


@functools.lru_cache(maxsize=1)
def _batch_scenes(items: int):
    """Small scenes of about 1 k to 100 k triangles; every fifth carries the medium sphere."""
    out = []
    for k in range(items):
        subdiv = 2 + k % 3
        sc = scenes.sphere_field(2 + (5 * k) % 17, subdiv, seed=1000 + k)
        if k % 5 == 4:
            sc.objects.append(scenes.medium_scene().objects[-1])
        out.append(sc)
    return out


def _context(sc):
    ctx = rx.Context(0)
    ctx.set_scene(sc)
    ctx.build_accel()
    return ctx


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _sphere(n, g):
    """Directions uniform on the sphere, (n, 3)."""
    u = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
    z = 1.0 - 2.0 * u[:, 0]
    s = (1.0 - z * z).clamp_min(0).sqrt()
    phi = 2.0 * math.pi * u[:, 1]
    return torch.stack([s * phi.cos(), s * phi.sin(), z], 1).float()


def _rays(n, seed):
    """rx_ray records: origins uniform in the room, directions uniform on the sphere."""
    g = _gen(seed)
    r = torch.zeros(n, 8, device="cuda")
    r[:, 0:3] = torch.rand(n, 3, generator=g, device="cuda") * ROOM
    r[:, 4:7] = _sphere(n, g)
    return r


def _records(n, seed):
    """Guiding records: position, normal, outgoing and incident directions, weight."""
    g = _gen(seed)
    r = torch.zeros(n, 16, device="cuda")
    r[:, 0:3] = torch.rand(n, 3, generator=g, device="cuda") * ROOM
    for k in (3, 6, 9):
        r[:, k:k + 3] = _sphere(n, g)
    r[:, 12] = -torch.rand(n, generator=g, device="cuda").clamp_min(1e-7).log()
    return r


def _weights(seed):
    """Network parameters of the size a trained network has, the layers' blocks in order."""
    rng = np.random.default_rng(seed)
    out = []
    for layer, k in enumerate(LAYERS):
        w = rng.standard_normal((64, k)) * math.sqrt(2.0 / k) * (0.5 if layer == 4 else 1.0)
        if layer == 4:
            w[40:] = 0.0
        out.append(w.reshape(-1))
    return np.concatenate(out).astype(np.float32)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed + 1)
    if kind in ("hit", "hit_host"):
        s["ctx"] = _context(_scene(case["spheres"], case["subdiv"]))
        n = case["rays"]
        rays = _rays(n, seed)
        if kind == "hit":
            s.update(rays=rays, tid=torch.empty(n, dtype=torch.int32, device="cuda"),
                     dist=torch.empty(n, dtype=torch.float32, device="cuda"))
        else:
            s.update(rays=rays.cpu().pin_memory().numpy(), tid=torch.empty(n, dtype=torch.int32).pin_memory().numpy(),
                     dist=torch.empty(n, dtype=torch.float32).pin_memory().numpy())
    elif kind in ("pt", "guided"):
        s["ctx"] = _context(_scene(case["spheres"], case["subdiv"]))
        s["camera"] = scenes.cornell_camera(case["width"], case["height"])
        if kind == "guided":
            s["ctx"].guide_init(train_passes=0, steps_per_pass=0, warmup_passes=0, box=BOX)
            s["ctx"].guide_set_params(_weights(seed))
    elif kind == "batch":
        cam = scenes.cornell_camera(case["res"], case["res"])
        s["items"] = [(_context(sc), cam, dict(spp=case["spp"], max_depth=case["depth"], rr_mode=1, nee=k % 2 == 1,
                                               seed=seed + k + 1))
                      for k, sc in enumerate(_batch_scenes(case["items"]))]
    elif kind in ("guide_eval", "guide_train"):
        n = case["rows"]
        s["ctx"] = rx.Context(0)
        s["ctx"].guide_init(batch=n, box=BOX)
        s["ctx"].guide_set_params(_weights(seed))
        s["recs"] = _records(n, seed)
        if kind == "guide_eval":
            s.update(raw=torch.empty(n, 40, device="cuda"), pdf=torch.empty(n, device="cuda"))
    else:
        sc = scenes.medium_scene(case["width"], case["height"])
        s["ctx"] = _context(sc)
        s["camera"] = sc.camera
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "hit":
        s["ctx"].trace_closest_device(s["rays"], case["rays"], s["tid"], s["dist"], stream=_stream())
        return s["tid"], s["dist"]
    if kind == "hit_host":
        s["ctx"].trace_closest_rays(s["rays"], s["tid"], s["dist"])
        return s["tid"], s["dist"]
    if kind in ("pt", "guided"):
        film, _, st = s["ctx"].render_pt(s["camera"], case["spp"], max_depth=case["depth"], rr_mode=1, seed=s["seed"],
                                         nee=bool(case.get("nee")), guided=kind == "guided")
        return film, st["extension_rays"], st["shadow_rays"]
    if kind == "batch":
        films, st = s["items"][0][0].render_pt_batch(s["items"])
        return films, st["extension_rays"], st["shadow_rays"]
    if kind == "guide_eval":
        s["ctx"].guide_eval_device(s["recs"], case["rows"], s["raw"], s["pdf"], stream=_stream())
        return s["raw"], s["pdf"]
    if kind == "guide_train":
        for _ in range(case["steps"]):
            s["ctx"].guide_train_step(s["recs"], case["rows"], stream=_stream(), want_loss=False)
        return s["ctx"].guide_params()
    if kind == "vcm":
        film, _ = s["ctx"].render_vcm(s["camera"], case["iterations"], 0.0963, 0.75, max_depth=case["depth"],
                                      light_paths=case["light_paths"], seed=s["seed"])
        return film
    film, _ = s["ctx"].render_bpt(s["camera"], case["iterations"], max_depth=case["depth"], seed=s["seed"])
    return film


# ---- what a pass cannot do without -------------------------------------------------------
def _triangles(case):
    return 36 + case["spheres"] * 20 * 4 ** case["subdiv"]


def _walk_flops(triangles):
    """One ray's walk at its least: a box test per level of a binary tree, two triangle tests."""
    return 18.0 * max(1.0, math.log2(triangles)) + 2 * 60.0


def work(case):
    kind = case["kind"]
    macs = 80 * 64 + 3 * 64 * 64 + 64 * 40
    if kind in ("hit", "hit_host"):
        t = _triangles(case)
        # rays in, answers out; the scene's triangles, at most as many as rays can touch
        return {"bytes": 40.0 * case["rays"] + 48.0 * min(t, case["rays"]), "flops": case["rays"] * _walk_flops(t)}
    if kind in ("pt", "guided"):
        t, px = _triangles(case), case["width"] * case["height"]
        paths = px * case["spp"]
        # about three bounces a path, each a ray and a scatter
        flops = 3.0 * paths * (_walk_flops(t) * (2 if case.get("nee") else 1) + 200.0)
        if kind == "guided":
            flops += 3.0 * paths * 2 * macs
        return {"bytes": 24.0 * px + 48.0 * min(t, 3 * paths), "flops": flops}
    if kind == "batch":
        px = case["items"] * case["res"] ** 2
        return {"bytes": 24.0 * px + 48.0 * 20_000 * case["items"],
                "flops": 3.0 * px * case["spp"] * (1.5 * _walk_flops(20_000) + 200.0)}
    if kind == "guide_eval":
        return {"bytes": case["rows"] * (64.0 + 164.0) + 86016.0, "flops": 2.0 * macs * case["rows"]}
    if kind == "guide_train":
        return {"bytes": case["steps"] * (case["rows"] * 64.0 + 7 * 86016.0),
                "flops": case["steps"] * 3 * 2.0 * macs * case["rows"]}
    px, t = case["width"] * case["height"], 36 + 20 * 4 ** 4
    light = case.get("light_paths", px)
    # both subpaths of about four vertices; for vcm the merges of the radius (about a
    # hundred photons a pixel and iteration at 2^20 light paths), each a join
    joins = px * (16.0 + (light / 2 ** 20 * 400.0 if kind == "vcm" else 0.0))
    return {"bytes": 24.0 * px, "flops": case["iterations"] * (4.0 * (px + light) * (_walk_flops(t) + 200.0) + joins * 300.0)}


# ---- the same in 64 bits -----------------------------------------------------------------
def _closest(case, seed):
    """Distance of the nearest triangle along each ray (-1: none), every triangle tried."""
    f = _scene(case["spheres"], case["subdiv"]).flatten()
    rays = _rays(case["rays"], seed).double()
    v = torch.from_numpy(f["verts"]).cuda().double()[torch.from_numpy(f["tris"].astype(np.int64)).cuda()]
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    out = []
    for r in rays.split(max(1, 40_000_000 // len(v0))):
        o, d = r[:, 0:3], r[:, 4:7]
        det = -(d @ nrm.T)
        # with a = o - v0: t = a.n / det, u = e2.(a x d) / det, w = -e1.(a x d) / det
        m = torch.linalg.cross(o, d)
        ad = lambda e: m @ e.T - d @ torch.linalg.cross(e, v0).T  # noqa: E731  (o - v0) x d . e
        t = (o @ nrm.T - (v0 * nrm).sum(1)) / det
        u, w = ad(e2) / det, -ad(e1) / det
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0)
        t = torch.where(ok, t, torch.inf).amin(1)
        out.append(torch.where(torch.isfinite(t), t, -1.0))
    return torch.cat(out)


def _network(params):
    out, at = [], 0
    for k in LAYERS:
        out.append(params[at:at + 64 * k].view(64, k))
        at += 64 * k
    return out


def _forward(params, recs):
    """The network's 40 outputs on the records, and the mixture's log density at wi."""
    p = recs[:, 0:3] / ROOM
    a = math.pi * 2.0 ** torch.arange(12, device="cuda", dtype=torch.float64) * p[:, :, None]
    x = torch.stack([a.sin(), a.cos()], -1).reshape(len(recs), 72)
    one = torch.ones(len(recs), 1, device="cuda", dtype=torch.float64)
    x = torch.cat([x, recs[:, 3:9], one, 0 * one], 1)
    w = _network(params)
    for k in range(4):
        x = (x @ w[k].T).relu()
    raw = (x @ w[4].T)[:, :40]
    lobe = raw.view(-1, 8, 5)
    kappa = lobe[..., 1].clamp(-4.0, 8.0).exp()
    mu = lobe[..., 2:5] / lobe[..., 2:5].norm(dim=-1, keepdim=True).clamp_min(1e-6)
    t = (mu * recs[:, None, 9:12]).sum(-1)
    norm = kappa.log() - math.log(2 * math.pi) - (-torch.expm1(-2 * kappa)).log()
    return raw, torch.logsumexp(lobe[..., 0].log_softmax(1) + norm + kappa * (t - 1.0), 1)


def _train(case, seed):
    """`steps` Adam steps on the records' weighted log-likelihood (weights clipped at 32 x their mean)."""
    params = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_()
    recs = _records(case["rows"], seed).double()
    w = recs[:, 12]
    w = w.clamp_max(32.0 * w.mean()) / w.sum()
    m, v = torch.zeros_like(params), torch.zeros_like(params)
    for t in range(1, case["steps"] + 1):
        grad = torch.zeros_like(params)
        for r, c in zip(recs.split(1 << 16), w.split(1 << 16)):
            grad += torch.autograd.grad(-(c * _forward(params, r)[1]).sum(), params)[0]
        with torch.no_grad():
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            params -= 5e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return params.detach()


def exact(case, seed):
    kind = case["kind"]
    if kind == "hit" and case["rays"] * _triangles(case) <= 4_000_000_000:
        return None, _closest(case, seed)
    if kind == "guide_eval":
        params, recs = torch.from_numpy(_weights(seed)).cuda().double(), _records(case["rows"], seed).double()
        got = [_forward(params, r) for r in recs.split(1 << 17)]
        return torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got]).exp()
    if kind == "guide_train":
        return _train(case, seed)
    return None
