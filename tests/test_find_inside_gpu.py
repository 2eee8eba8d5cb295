"""find_inside through the library, with media that nest and overlap. The camera sits in two
absorbing media at once (no scattering, no refraction) inside a room of constant emission:
the last-listed medium around it is the one its rays start in. A camera ray that meets the
other one's surface first ends there (a medium within a medium is not modelled); else it
leaves through the first one's own surface into the other, if the leaving point lies in it,
and through that one's into the room, where a third medium may lie in its way. Each pixel's
expectation follows from the distances at which its rays cross the meshes (every triangle
tried, double precision). Near the origin and hundreds of units away from it."""
import functools

import numpy as np
import pytest

import renderx_gb300 as rx
from renderx_gb300 import scenes
from renderx_gb300.scenes import EMISSIVE, VPM, Camera, Material, Obj, Scene

pytestmark = pytest.mark.gpu
N, SPP, SUB = 16, 8192, 8
SIGMA = {"a": np.array([0.9, 0.5, 0.2]), "b": np.array([0.1, 0.6, 1.1]), "far": np.array([3.0, 3.0, 3.0])}
PLACES = {  # centre and radius of each medium, camera
    "nested": ({"a": ((0, 0, 0), 2.0), "b": ((0.3, 0.2, -0.1), 0.8), "far": ((4.0, 3.0, -4.0), 0.7)}, (0.1, 0.3, 0.1)),
    "overlapping": ({"a": ((0, 0, 0), 1.5), "b": ((1.1, 0.2, 0), 1.3), "far": ((-4.0, 3.0, 4.0), 0.7)}, (0.5, 0.1, 0.2)),
}


def crossings(o, d, verts, tris):
    """Distances of the first and the last crossing of the mesh by the ray from o along each d
    (infinite and -infinite where there is none)."""
    v = verts.astype(np.float64)[tris]
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    first, last = np.full(len(d), np.inf), np.full(len(d), -np.inf)
    for k in range(0, len(d), 1024):
        dd = d[k:k + 1024, None]
        p = np.cross(dd, e2[None])
        with np.errstate(all="ignore"):
            inv = 1.0 / np.sum(e1 * p, -1)
            s = o - v0
            u = np.sum(s * p, -1) * inv
            q = np.cross(s, e1)
            w = np.sum(dd * q[None], -1) * inv
            t = np.sum(e2 * q, -1) * inv
            hit = (u >= -1e-9) & (w >= -1e-9) & (u + w <= 1 + 1e-9) & (t > 0)
        first[k:k + 1024] = np.where(hit, t, np.inf).min(1)
        last[k:k + 1024] = np.where(hit, t, -np.inf).max(1)
    return first, last


def passed(sigma, dist):
    """Expectation of a path's weight over `dist` in a medium: the transmittance, over the density
    of passing that the estimator divides by (the luminance of the transmittance), times the
    probability of passing with which it samples (by the luminance of the extinction)."""
    lum = np.array([0.212671, 0.715160, 0.072169])
    t = np.exp(-dist[:, None] * sigma)
    return t * (np.exp(-dist * (lum @ sigma)) / (t @ lum))[:, None]


@functools.lru_cache(maxsize=None)
def setting(place, offset):
    """Meshes, camera, and the crossings of each mesh by the rays of a grid in every pixel."""
    media, cam = PLACES[place]
    off = np.asarray(offset)
    uv, uf = scenes.icosphere(3)
    tris = uf.astype(np.uint32)
    mesh = {k: (off + np.asarray(c) + r * uv).astype(np.float32) for k, (c, r) in media.items()}
    pos = (np.asarray(cam) + off).astype(np.float32)
    camera = Camera(N, N, 3 * N // 4, tuple(pos.tolist()), tuple((pos + np.float32([0.5, 0.25, -1.0])).tolist()))
    front = np.asarray(camera.focus, np.float64) - np.asarray(camera.position)
    front /= np.linalg.norm(front)
    right = np.cross(front, camera.up)
    right /= np.linalg.norm(right)
    up = np.cross(right, front)
    g = (np.arange(N * SUB) + 0.5) / SUB
    y, x = np.meshgrid(g, g, indexing="ij")
    d = front * camera.sight_dist + right * (x - N / 2)[..., None] + up * (N / 2 - y)[..., None]
    d = (d / np.linalg.norm(d, axis=-1, keepdims=True)).reshape(-1, 3)
    return mesh, tris, camera, {k: crossings(pos.astype(np.float64), d, mesh[k], tris) for k in media}


@pytest.mark.parametrize("offset", [(0.0, 0.0, 0.0), (800.0, -300.0, 50.0)])
@pytest.mark.parametrize("order", [("far", "a", "b"), ("b", "a", "far"), ("b", "far", "a")])
@pytest.mark.parametrize("place", ["nested", "overlapping"])
def test_rays_start_and_go_on_in_the_right_medium(place, order, offset):
    mesh, tris, camera, t = setting(place, offset)
    bv, bt = scenes._box((0.0, 0.0, 0.0), (14.0, 14.0, 14.0), 0.0)
    room = Obj("room", (bv + np.asarray(offset)).astype(np.float32), np.ascontiguousarray(bt[:, ::-1]),
               Material(EMISSIVE, (1.0, 1.0, 1.0)))
    balls = [Obj(k, mesh[k], tris, Material(VPM, (1.0, 1.0, 1.0), ior=1.0, sigma_a=tuple(SIGMA[k]))) for k in order]
    films = []
    for objects in ([room], [room, *balls]):
        with rx.Context(0) as c:
            c.set_scene(Scene(objects, camera))
            c.build_accel()
            film, sq, _ = c.render_pt(camera, SPP, max_depth=8, seed=11, want_sq=True)
            films.append((film, sq))
    first, then = ("b", "a") if order.index("b") > order.index("a") else ("a", "b")
    t1, t2 = t[first][0], t[then][0]
    assert np.isfinite(t1).all() and np.isfinite(t2).all()
    ends, far = t2 < t1, np.isfinite(t["far"][0])
    weight = passed(SIGMA[first], t1) * passed(SIGMA[then], np.maximum(t2 - t1, 0.0))
    weight *= passed(SIGMA["far"], np.where(far, t["far"][1] - t["far"][0], 0.0))
    weight[ends] = 0.0
    pixels = lambda a: a.reshape(N, SUB, N, SUB, -1)  # noqa: E731
    want = pixels(weight).mean((1, 3)) * films[0][0]
    # pixels whose rays all cross the same surfaces: the grid's rays and those of the pixels
    # around them do (a sliver at a pixel's corner passes between the grid's rays)
    whole = np.ones((N, N), bool)
    for m in (ends, t2 > t1, far):
        share = np.pad(pixels(m).mean((1, 3))[..., 0], 1, mode="edge")
        near = np.lib.stride_tricks.sliding_window_view(share, (3, 3)).reshape(N, N, 9)
        whole &= (near == 0.0).all(-1) | (near == 1.0).all(-1)
    film, sq = films[1]
    se = np.sqrt(np.maximum(sq - film * film, 0.0) / (SPP - 1))
    # the sub-pixel grid and the single-precision distances (1e-4 of a unit at 800) are far below
    # a standard error of a hundredth of the value
    z = (np.abs(film - want) / (se + 2e-4 * want + 1e-12))[whole]
    assert whole.mean() > 0.6 and (z > 3).mean() <= 0.02 and z.max() < 6, (whole.mean(), (z > 3).mean(), z.max())
    if place == "overlapping":  # both kinds of ray
        assert (want[whole].sum(-1) == 0.0).sum() > 40 and (want[whole].sum(-1) > 0.0).sum() > 40
