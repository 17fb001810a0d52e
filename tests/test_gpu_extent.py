"""Scenes much larger than their detail: 20000 triangles of 0.02 on a ground from -half to half.
The ground must not cost the detail its hierarchy, and a ray that comes from as far as the ground
reaches must still find what it hits."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def detail(rg, half, n=20000):
    rng = np.random.default_rng(1)
    c = rng.uniform(-2, 2, (n, 1, 3)) * [1, 0.4, 1] + [0, -0.2, -6]
    pos = (c + rng.normal(size=(n, 3, 3)) * 0.01).astype(np.float32).reshape(n, 9)
    up = np.tile(np.array([0, 1, 0], np.float32), 3)
    a, b = (-half, -1.2, -half), (half, -1.2, half)
    ground = np.array([a + (half, -1.2, -half) + b, a + b + (-half, -1.2, half)], np.float32)
    return scenes.build(rg, [(pos, np.tile(up, (n, 1)), scenes.material(rg), -1),
                             (ground, np.tile(up, (2, 1)), scenes.material(rg), -1)], scenes.camera(rg)), pos


def renderer(rg, scene):
    r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=64, resolutionHeight=48, samples=2, maxDepth=4))
    r.set_scene(scene)
    return r


@pytest.mark.parametrize("half", [1e4, 1e5, 1e6])
def test_work_per_ray_does_not_grow_with_the_ground(rg, half):
    per_ray = []
    for h in (10.0, half):
        scene, _ = detail(rg, h)
        r = renderer(rg, scene)
        r.render()
        s = r.stats()
        per_ray.append(((s["nodes_visited"] + s["tris_tested"]) / s["closest_rays"]))
        r.close()
        scene.close()
    # the far ground's hits add rays that leave the detail alone, never more work than half as much again
    assert per_ray[1] < 1.5 * per_ray[0]


def clear_hits(pos, rays):
    """Per ray the nearest of the triangles that it hits so far from their edges that the FP32
    triangle test finds them too, in 64 bits (infinity: none)."""
    v = pos.reshape(-1, 3, 3).astype(np.float64)
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    size = np.maximum(np.linalg.norm(e1, axis=1), np.linalg.norm(e2, axis=1))
    out = np.full(len(rays), np.inf)
    for i, r in enumerate(rays.astype(np.float64)):
        o, d = r[:3], r[3:]
        p = np.cross(d, e2)
        det = (e1 * p).sum(1)
        s = o - v0
        q = np.cross(s, e1)
        with np.errstate(divide="ignore", invalid="ignore"):
            u, w, t = (s * p).sum(1) / det, q @ d / det, (e2 * q).sum(1) / det
            # rounding of o - v0 and of the products after it, as a part of the triangle
            m = 16 * 2.0 ** -24 * np.linalg.norm(s, axis=1) * size / np.abs(det) + 1e-3
        ok = (np.abs(det) > 1e-5) & (u > m) & (w > m) & (u + w < 1 - m) & (t > 1e-3)
        out[i] = t[ok].min(initial=np.inf)
    return out


@pytest.mark.parametrize("half", [10.0, 1e3, 1e4])
@pytest.mark.parametrize("copies", [1, 40])  # a warp per ray, and a lane per ray
def test_rays_from_afar_miss_nothing(rg, half, copies):
    scene, pos = detail(rg, half, 4000)
    n = 1000
    rng = np.random.default_rng(3)
    target = pos.reshape(-1, 3, 3)[rng.integers(0, len(pos), n)].mean(1)
    d = rng.normal(size=(n, 3)) * [1, 0.2, 1]
    d[::7] = np.eye(3)[rng.integers(0, 3, len(d[::7]))]  # along the axes
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = target - d * np.exp(rng.uniform(np.log(0.5), np.log(half), (n, 1)))
    rays = np.concatenate([o, d], axis=1).astype(np.float32)
    t = clear_hits(pos, rays)
    clear = np.isfinite(t)
    assert clear.sum() > 300
    r = renderer(rg, scene)
    got = r.trace_closest(np.tile(rays, (copies, 1)))[0][:, 0].reshape(copies, n)
    occluded = r.trace_any(np.tile(rays, (copies, 1)), np.full(copies * n, 4 * half, np.float32)).reshape(copies, n)
    r.close()
    scene.close()
    # a distance is off by up to 8 x 2^-24 size^2 / det of itself: 4e-5 at the thinnest that count
    assert (got[:, clear] <= t[clear] * (1 + 1e-4)).all()
    assert (occluded[:, clear] == 1).all()
