"""The bounds rule of find_inside (renderx_gb300/csrc/rx_material.cuh): a point outside a
medium's padded bounds is never inside the medium, and every hit that decides lies before
the ray leaves the bounds. The reference's test (both the +d and -d rays leave the object
through its surface, reference src/Scene.cpp:354-390) is restated in float32 over every
triangle and compared with the rule on points around, on and inside spheres of several
sizes and places."""
import numpy as np
import pytest

from renderx_gb300 import scenes


def leaves(o, d, v0, e1, e2, nrm):
    """Per point: whether the ray leaves the object, and its distance (float32)."""
    pv = np.cross(d[:, None], e2[None])
    with np.errstate(all="ignore"):
        det = np.sum(e1[None] * pv, -1)
        sv = o[:, None] - v0[None]
        u = np.sum(sv * pv, -1) / det
        qv = np.cross(sv, e1[None])
        v = np.sum(d[:, None] * qv, -1) / det
        t = np.sum(e2[None] * qv, -1) / det
        ok = (np.abs(det) >= 1e-30) & (u >= -1e-7) & (u <= 1.0000001) & (v >= -1e-7) & (u + v <= 1.0000001) & (t >= 0)
    t = np.where(ok, t, np.inf)
    k = t.argmin(1)
    t = t[np.arange(len(o)), k]
    return np.isfinite(t) & (t >= 1e-6) & (np.sum(nrm[k] * d, 1) >= 1e-6), t


@pytest.mark.parametrize("centre,radius", [((2.78, 3.0, 1.5), 1.0), ((0.0, 0.0, 0.0), 1e-3), ((800.0, -300.0, 50.0), 2.0)])
def test_points_outside_the_padded_bounds_are_not_inside(centre, radius):
    rng = np.random.default_rng(5)
    uv, uf = scenes.icosphere(2)
    verts = (np.asarray(centre) + radius * uv).astype(np.float32)
    v0, v1, v2 = (verts[uf[:, k]] for k in range(3))
    e1, e2 = v1 - v0, v2 - v0
    nrm = np.cross(e1, e2)
    nrm = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    lo, hi = verts.min(0), verts.max(0)
    pad = np.float32(max(1e-3 * (hi[a] - lo[a]) + 1e-4 * max(abs(lo[a]), abs(hi[a])) + 1e-5 for a in range(3)))
    lo, hi = lo - pad, hi + pad
    n = 20000
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    # a third on the surface (where boundary scatters start), the others in a box 1.5 times as wide
    on = rng.integers(0, len(uf), n // 3)
    b = rng.dirichlet((1, 1, 1), n // 3)[:, :, None].astype(np.float32)
    o = np.concatenate([b[:, 0] * v0[on] + b[:, 1] * v1[on] + b[:, 2] * v2[on],
                        np.asarray(centre) + radius * rng.uniform(-1.5, 1.5, (n - n // 3, 3))]).astype(np.float32)
    inside = np.ones(n, bool)
    for dd in (-d, d):
        out, t = leaves(o, dd, v0, e1, e2, nrm.astype(np.float32))
        with np.errstate(all="ignore"):
            inv = np.where(np.abs(dd) > 1e-30, 1 / dd, np.copysign(1e30, dd)).astype(np.float32)
            tmax = np.where(inv < 0, (lo - o) * inv, (hi - o) * inv).min(1)
        in_box = ((o >= lo) & (o <= hi)).all(1)
        assert (t[out & in_box] < tmax[out & in_box]).all()
        inside &= out
    assert inside.sum() > 500
    assert in_box[inside].all()
