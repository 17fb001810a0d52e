"""BVH builds at the edges of the block-wise subtree pass (1024 primitives) and of the
device-wide levels: triangle counts around the limits, spread, clustered (unbalanced trees)
and with coincident centroids (median splits).  Hits must equal those of the general build
(more than 32 bins: device-wide levels down to the leaves) and of a brute-force scan, since a
triangle's test does not depend on the tree; distances are compared exactly between builds,
and triangles except where distances tie."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def triangles(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "coincident":
        c = np.zeros((n, 1, 3))
    elif kind == "clustered":  # exponentially shrinking clusters
        c = rng.normal(size=(n, 1, 3)) * np.exp(-rng.uniform(0, 9, (n, 1, 1)))
    elif kind == "flat":
        c = rng.uniform(-2, 2, (n, 1, 3)) * np.array([1.0, 1.0, 0.0])
    else:
        c = rng.uniform(-2, 2, (n, 1, 3))
    size = 0.3 / np.sqrt(max(n, 4)) * 8
    e = rng.normal(size=(n, 3, 3)) * size
    if kind == "coincident":
        e -= e.mean(axis=1, keepdims=True)
    return (c + e + np.array([0, 0, -6.0])).astype(np.float32).reshape(n, 9)


def scene_of(rg, pos):
    nrm = np.tile(np.array([0, 0, 1], np.float32), (len(pos), 3))
    return scenes.build(rg, [(pos, nrm, scenes.material(rg), -1)], scenes.camera(rg))


def hits(rg, scene, rays, bins, width):
    r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=8, resolutionHeight=8, samples=1, bvhBins=bins, bvhWidth=width))
    r.set_scene(scene)
    tuv, prim = r.trace_closest(rays)
    occ = r.trace_any(rays, np.full(len(rays), 6.0, np.float32), rg.PRED_ALL)
    r.close()
    return tuv, prim, occ


@pytest.mark.parametrize("kind", ["spread", "clustered", "coincident", "flat"])
@pytest.mark.parametrize("n", [1, 4, 5, 9, 1023, 1024, 1025, 2051, 9000])
def test_builds_agree(rg, kind, n):
    pos = triangles(kind, n, n)
    scene = scene_of(rg, pos)
    rng = np.random.default_rng(n + 1)
    k = 3000
    o = np.concatenate([np.zeros((k // 2, 3)), rng.uniform(-3, 3, (k - k // 2, 3)) + [0, 0, -3.0]])
    target = pos.reshape(-1, 3, 3).mean(1)[rng.integers(0, n, k)] + rng.normal(size=(k, 3)) * 0.05
    rays = np.concatenate([o, target - o], axis=1).astype(np.float32)
    tuv, prim, occ = hits(rg, scene, rays, 32, 8)
    assert (prim >= 0).any()
    for bins, width in [(48, 8), (32, 2), (17, 8), (48, 2)]:
        t2, p2, o2 = hits(rg, scene, rays, bins, width)
        np.testing.assert_array_equal(tuv[:, 0], t2[:, 0])
        np.testing.assert_array_equal(occ, o2)
        assert (prim != p2).mean() < 0.002  # equal distances only
    # brute force in 64 bits for a few rays: no triangle is missing from the tree
    sub = slice(0, 200)
    t = np.full(200, np.inf)
    d, s = rays[sub, 3:].astype(np.float64), rays[sub, :3].astype(np.float64)
    for tri in pos.reshape(-1, 3, 3).astype(np.float64):
        e1, e2 = tri[1] - tri[0], tri[2] - tri[0]
        p = np.cross(d, e2)
        det = p @ e1
        with np.errstate(divide="ignore", invalid="ignore"):
            u = ((s - tri[0]) * p).sum(1) / det
            q = np.cross(s - tri[0], e1)
            v, tt = (d * q).sum(1) / det, q @ e2 / det
        inside = (np.abs(det) > 1e-7) & (u > 1e-4) & (v > 1e-4) & (u + v < 1 - 1e-4) & (tt > 1e-4)
        t = np.where(inside, np.minimum(t, tt), t)
    clear = np.isfinite(t)
    assert (tuv[sub, 0][clear] <= t[clear] * (1 + 1e-4)).all()
    scene.close()
