"""The 8-wide traversal kernels at the edges of their warp-wide triangle queue.

Transparent quads stacked along the view: every ray hits every layer's triangles, so a node
hands a lane up to 32 of them at once.  Few pixels leave warps with few rays (triangles go
through the queue, which then overflows and drains), many fill them (lanes test their own).
The image must equal the binary BVH's, whose kernels test triangles one by one: the triangle
test is the same arithmetic, and no two layers lie at the same distance.
"""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def stacked(rg, layers):
    parts = []
    for k in range(layers):
        p, n = scenes.quad_z(-2.0 - 0.05 * k, 3.0, +1)
        parts.append((p, n, scenes.material(rg, (0.9, 0.8, 0.7), transparency=0.6), -1))
    p, n = scenes.quad_z(-2.0 - 0.05 * layers - 1.0, 6.0, +1)
    parts.append((p, n, scenes.material(rg, (0.5, 0.6, 0.7)), -1))
    p, n = scenes.quad_z(1.5, 2.0, -1)
    parts.append((p, n, scenes.material(rg, (1, 1, 1), emission=4.0), -1))
    return scenes.build(rg, parts, scenes.camera(rg, fov=50.0))


def image(rg, scene, w, h, spp, width):
    r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=w, resolutionHeight=h, samples=spp, maxDepth=8, seed=3,
                                           bvhWidth=width))
    r.set_scene(scene)
    r.render()
    out = r.get_hdr_result()
    r.close()
    return out


@pytest.mark.parametrize("layers", [1, 4, 15, 16, 17, 70])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (5, 1, 1), (11, 1, 1), (12, 1, 1), (33, 1, 1), (65, 9, 2)])
def test_stacked_layers_equal_the_binary_bvh(rg, layers, w, h, spp):
    scene = stacked(rg, layers)
    np.testing.assert_array_equal(image(rg, scene, w, h, spp, 8), image(rg, scene, w, h, spp, 2))
    scene.close()


@pytest.mark.parametrize("w,h", [(3, 1), (11, 1), (40, 30)])
def test_equal_distances_do_not_depend_on_the_warp(rg, w, h):
    """Coincident quads of other colours and orders: every ray has exact ties.  The triangle
    found first is the hit, however many rays a warp holds and in which order its queue and its
    lanes test triangles: waves of one path give the image of full waves."""
    rng = np.random.default_rng(4)
    parts = []
    for k in range(24):
        p, n = scenes.quad_z(-2.0 - 0.1 * (k // 6), 3.0, +1)
        color = tuple(rng.uniform(0.2, 0.9, 3))
        parts.append((p, n, scenes.material(rg, color, transparency=0.5 if k < 18 else 0.0), -1))
    p, n = scenes.quad_z(1.5, 2.0, -1)
    parts.append((p, n, scenes.material(rg, (1, 1, 1), emission=4.0), -1))
    scene = scenes.build(rg, parts, scenes.camera(rg, fov=50.0))
    images = []
    for paths in (0, 1 if w * h < 50 else 37):
        r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=w, resolutionHeight=h, samples=2, maxDepth=8, seed=5,
                                               pathsPerWave=paths))
        r.set_scene(scene)
        r.render()
        images.append(r.get_hdr_result())
        r.close()
    np.testing.assert_allclose(images[0], images[1], rtol=1e-6)  # sums of two samples, grouped by wave
    scene.close()
