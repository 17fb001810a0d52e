"""BVH builds over triangles that are no numbers or whose boxes' areas overflow, at every size of
the device-wide levels and of the block-wise subtrees.

A split whose cost is no number (0 x infinity) leaves a warp's lanes with different choices; the
build must refuse such a node or take one lane's choice, and the handle stays usable either way."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def spread(n, seed=5):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-2, 2, (n, 1, 3)) + np.array([0, 0, -6.0])
    return (c + rng.normal(size=(n, 3, 3)) * 0.1).astype(np.float32).reshape(n, 9)


def scene_of(rg, pos):
    nrm = np.tile(np.array([0, 0, 1] * 3, np.float32), (len(pos), 1))
    return scenes.build(rg, [(pos, nrm, scenes.material(rg), -1)], scenes.camera(rg))


def renderer(rg, width=8, bins=32):
    return rg.RayRenderer(rg.RendererSettings(resolutionWidth=8, resolutionHeight=8, samples=1, bvhWidth=width, bvhBins=bins))


def still_works(rg, r, n):
    pos = spread(n, 9)
    scene = scene_of(rg, pos)
    target = pos.reshape(-1, 3, 3).mean(1)[:200]
    rays = np.concatenate([np.zeros_like(target), target], axis=1).astype(np.float32)
    r.set_scene(scene)
    got = r.trace_closest(rays)
    other = renderer(rg, bins=48)
    other.set_scene(scene)
    want = other.trace_closest(rays)
    other.close()
    scene.close()
    assert (got[1] >= 0).all()
    np.testing.assert_array_equal(got[0][:, 0], want[0][:, 0])


@pytest.mark.parametrize("width,bins", [(8, 32), (2, 32), (8, 48)])
@pytest.mark.parametrize("n", [1, 4, 5, 8, 9, 300, 1024, 1025, 5000])
def test_a_triangle_of_nan(rg, width, bins, n):
    """Accepted or refused, by how the bounds' integer form orders a NaN, which nothing promises."""
    pos = spread(n)
    pos[n // 2] = np.nan
    scene = scene_of(rg, pos)
    r = renderer(rg, width, bins)
    try:
        r.set_scene(scene)
    except rg.RayGenError as e:
        assert "scatter" in str(e)
    scene.close()
    still_works(rg, r, max(n, 20))
    r.close()


@pytest.mark.parametrize("n", [9, 700, 1500])
@pytest.mark.parametrize("far", [1e20, -1e20])
def test_areas_that_overflow(rg, n, far):
    """One triangle far out: its own area and the root's are infinite, so every split costs 0 x inf."""
    pos = spread(n)
    pos[0] = np.float32(far) * np.array([1, 1, 1, 2, 1, 1, 1, 2, 1], np.float32)
    scene = scene_of(rg, pos)
    r = renderer(rg)
    with pytest.raises(rg.RayGenError, match="scatter"):
        r.set_scene(scene)
    scene.close()
    still_works(rg, r, n)
    r.close()


@pytest.mark.parametrize("n", [9, 700, 1500])
def test_an_infinite_vertex(rg, n):
    """An infinite extent puts every primitive into bin 0: halves by index, accepted."""
    pos = spread(n)
    pos[0, 0] = np.inf
    scene = scene_of(rg, pos)
    r = renderer(rg)
    r.set_scene(scene)
    scene.close()
    still_works(rg, r, n)
    r.close()
